"""Products whose dictionaries or weights the tensor maps do not take: fp32 throughout, at the edges
of the kernel's tiles, against 64-bit products of the oracle's weight."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu

# Sums of `cols` products of 24-bit operands in fp32, in blocks: the relative error stays below
# sqrt(cols) * 2^-24, 7e-6 at 11008; 4e-6 leaves what is measured (below 6e-7) a wide margin.
FP32 = 4e-6


def product(ctx, pay, x, dtype, token, bias=None):
    seg = cs.Segment.from_payload(pay, ctx)
    m = x.shape[0]
    t = torch.from_numpy(x).cuda()
    t = t.bfloat16() if dtype == "bf16" else t
    xin = t.contiguous() if token else t.t().contiguous()
    y = torch.full((m, seg.rows) if token else (seg.rows, m), float("nan"), device="cuda")
    b = torch.from_numpy(bias).cuda() if bias is not None else None
    torch.cuda.synchronize()
    layout = cs.TOKEN_MAJOR if token else cs.FEATURE_MAJOR
    for _ in range(2):
        seg.matmul_device(xin.data_ptr(), cs.DTYPE_BF16 if dtype == "bf16" else cs.DTYPE_F32, layout, m, y.data_ptr(), layout,
                          b.data_ptr() if b is not None else 0)
    ctx.synchronize()
    return (y if token else y.t()).double().cpu().numpy(), t.double().cpu().numpy()


@pytest.mark.parametrize("token", [False, True])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows,cols,tile,atoms,k,m", [
    (70, 31, 0, 10, 3, 1),          # narrower than a block of columns
    (65, 97, 0, 65, 8, 2),          # one row past a row tile, odd width
    (300, 1021, 0, 300, 8, 5),      # column ranges, odd width
    (300, 1024, 0, 300, 5, 16),     # aligned rows, widest narrow tile
    (129, 514, 0, 128, 8, 17),      # one token past the narrow tile; width 2 mod 4
    (90, 2050, 0, 100, 8, 32),      # the middle token tile exactly, several blocks a range
    (64, 1000, 0, 129, 4, 64),      # a token tile exactly
    (513, 333, 0, 40, 8, 131),      # ragged in every direction
    (100, 100, 16, 20, 4, 3),       # tiles with both strips, few tokens
    (131, 259, 32, 24, 8, 40),
    (256, 260, 32, 24, 5, 70),      # bottom-aligned, strip on the right
])
def test_fp32_products(ctx, oracle, rows, cols, tile, atoms, k, m, dtype, token):
    tr, tc = (tile, tile) if tile else (1, cols)
    pay = synth.hsdr_payload(rows, cols, tile_rows=tr, tile_cols=tc, n_atoms=atoms, k=k, seed=rows * 3 + cols)
    rng = np.random.default_rng(m)
    x, bias = rng.normal(0, 1, (m, cols)).astype(np.float32), rng.normal(0, 1, rows).astype(np.float32)
    got, xd = product(ctx, pay, x, dtype, token, bias)
    want = xd @ oracle.decompress(pay).astype(np.float64).T + bias
    assert np.linalg.norm(got - want) <= FP32 * np.linalg.norm(want)


@pytest.mark.parametrize("members,cols,m", [(3, 97, 3), (5, 97, 16), (2, 1024, 40), (18, 33, 1)])
def test_groups_of_fp32_products(ctx, oracle, members, cols, m):
    """One activation, members of 10 to 78 atoms (projections off 16-byte steps), more than a gather
    launch or a projection launch holds."""
    pays = [synth.hsdr_payload(50 + 7 * i, cols, n_atoms=10 + 4 * i + i % 3, k=3 + i % 4, seed=i) for i in range(members)]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    x = torch.from_numpy(np.random.default_rng(m).normal(0, 1, (m, cols)).astype(np.float32)).cuda()
    ys = [torch.full((m, s.rows), float("nan"), device="cuda") for s in segs]
    torch.cuda.synchronize()
    cs.Segment.matmul_group_device(segs, x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, [y.data_ptr() for y in ys], cs.TOKEN_MAJOR)
    ctx.synchronize()
    xd = x.double().cpu().numpy()
    for pay, y in zip(pays, ys):
        want = xd @ oracle.decompress(pay).astype(np.float64).T
        assert np.linalg.norm(y.double().cpu().numpy() - want) <= FP32 * np.linalg.norm(want)


def test_lists_of_odd_width(ctx, oracle):
    """Independent products share launches; one that reads another's result comes behind it; a different
    width or form starts anew."""
    rng = np.random.default_rng(5)
    shapes = [(31, 45), (64, 45), (45, 31), (77, 45), (20, 99), (33, 99)]     # the third reads the first's result
    pays = [synth.hsdr_payload(r, c, n_atoms=20, k=4, seed=r + c) for r, c in shapes]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    xs = [torch.from_numpy(rng.normal(0, 1, (2, c)).astype(np.float32)).cuda() for _, c in shapes]
    ys = [torch.full((2, r), float("nan"), device="cuda") for r, _ in shapes]
    xs[2] = ys[0]
    torch.cuda.synchronize()
    cs.Segment.matmul_queue_device([(s, x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, 2, y.data_ptr(), cs.TOKEN_MAJOR, 0, 0 if i == 2 else -1)
                                    for i, (s, x, y) in enumerate(zip(segs, xs, ys))])
    ctx.synchronize()
    for pay, x, y in zip(pays, xs, ys):
        want = x.double().cpu().numpy() @ oracle.decompress(pay).astype(np.float64).T
        assert np.linalg.norm(y.double().cpu().numpy() - want) <= FP32 * np.linalg.norm(want)

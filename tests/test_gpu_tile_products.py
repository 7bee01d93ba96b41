"""2-D tiles on the tensor cores: the tile products of a few tokens (one CTA walking many row tiles,
one to three column blocks, several token tiles) and the wide products written token-major, against
64-bit products of the oracle's weight."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu

# Operands split into two bf16 pieces leave 2^-17 of every product; the rest is the tensor cores'
# fp32 accumulation over at most 512 columns.
SPLIT = 2e-5


def product(ctx, pay, x, dtype, token, shift=0):
    seg = cs.Segment.from_payload(pay, ctx)
    m = x.shape[0]
    t = torch.from_numpy(x).cuda()
    t = t.bfloat16() if dtype == "bf16" else t
    xin = t.contiguous() if token else t.t().contiguous()
    room = torch.full((m * seg.rows + shift,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    layout = cs.TOKEN_MAJOR if token else cs.FEATURE_MAJOR
    for _ in range(2):
        seg.matmul_device(xin.data_ptr(), cs.DTYPE_BF16 if dtype == "bf16" else cs.DTYPE_F32, layout, m, room.data_ptr() + 4 * shift, layout)
    ctx.synchronize()
    y = room[shift:].view((m, seg.rows) if token else (seg.rows, m))
    return (y if token else y.t()).double().cpu().numpy(), t.double().cpu().numpy()


@pytest.mark.parametrize("token", [False, True])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows,cols,tr,tc,atoms,k,m", [
    (128, 64, 32, 8, 4, 4, 1),            # one row tile of products, eight tokens of eight columns
    (256, 240, 64, 24, 10, 5, 3),         # five row tiles, part of a column block
    (256, 512, 128, 128, 160, 8, 2),      # more row tiles than SMs: both accumulators in turn
    (128, 408, 128, 136, 20, 8, 3),       # three column blocks, the last one partly outside
    (256, 512, 32, 32, 16, 4, 15),        # 240 tokens: two token tiles, the second partly outside
    (128, 384, 128, 128, 160, 8, 13),     # 39 tokens in a tile of 48
    (128, 576, 32, 32, 20, 4, 8),         # 144 tokens in two tiles of 80
])
def test_tile_products(ctx, oracle, rows, cols, tr, tc, atoms, k, m, dtype, token):
    pay = synth.hsdr_payload(rows, cols, tile_rows=tr, tile_cols=tc, n_atoms=atoms, k=k, seed=rows + tc)
    x = np.random.default_rng(m).normal(0, 1, (m, cols)).astype(np.float32)
    got, xd = product(ctx, pay, x, dtype, token)
    want = xd @ oracle.decompress(pay).astype(np.float64).T
    assert np.linalg.norm(got - want) <= SPLIT * np.linalg.norm(want)


@pytest.mark.parametrize("shift", [0, 1])      # 1: results off 16-byte boundaries
@pytest.mark.parametrize("rows,cols,m", [(128, 256, 16), (256, 264, 37), (512, 128, 64), (19072, 64, 16)])
def test_wide_products_token_major(ctx, oracle, rows, cols, m, shift):
    pay = synth.hsdr_payload(rows, cols, tile_rows=32, tile_cols=8, n_atoms=16, k=4, seed=rows + cols)
    x = np.random.default_rng(m).normal(0, 1, (m, cols)).astype(np.float32)
    got, xd = product(ctx, pay, x, "f32", True, shift)
    want = xd @ oracle.decompress(pay).astype(np.float64).T
    assert np.linalg.norm(got - want) <= SPLIT * np.linalg.norm(want)


@pytest.mark.parametrize("m", [3, 7, 11, 15])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_chunks_of_three_tokens(oracle, dtype, m):
    """The gather's last chunk holds three tokens in a place for four; the products of the fourth would
    lie behind the tile products (10 MB a chunk, in a context that has no larger scratch)."""
    ctx = cs.Context(0)
    pay = synth.hsdr_payload(640, 1664, tile_rows=128, tile_cols=128, n_atoms=512, k=5, seed=m)
    x = np.random.default_rng(m).normal(0, 1, (m, 1664)).astype(np.float32)
    got, xd = product(ctx, pay, x, dtype, True)
    want = xd @ oracle.decompress(pay).astype(np.float64).T
    assert np.linalg.norm(got - want) <= SPLIT * np.linalg.norm(want)
    ctx.close()

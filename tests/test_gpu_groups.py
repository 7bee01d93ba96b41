"""Groups on the one-launch GEMV: the members' projections handed over and their rows walked together
where their slices fit shared memory, one member after the other where not; members of unequal rows
(some CTAs without rows of one), atoms and codes."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("cols,members", [
    (64, [(3, 10, 8), (5, 16, 3)]),                          # fewer rows than CTAs
    (900, [(896, 512, 8), (128, 128, 5), (128, 300, 8)]),    # one column range
    (2052, [(5000, 96, 8), (40, 512, 4)]),                   # three column ranges, rows far apart
    (1024, [(300, 4000, 8), (200, 3000, 8), (100, 2000, 8)]),  # slices past what fits: one after the other
])
def test_groups(ctx, oracle, cols, members, m):
    pays = [synth.hsdr_payload(r, cols, n_atoms=a, k=k, seed=r + a) for r, a, k in members]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    x = torch.from_numpy(np.random.default_rng(m).normal(0, 1, (m, cols)).astype(np.float32)).cuda()
    ys = [torch.full((m, s.rows), float("nan"), device="cuda") for s in segs]
    torch.cuda.synchronize()
    for _ in range(3):
        cs.Segment.matmul_group_device(segs, x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, [y.data_ptr() for y in ys], cs.TOKEN_MAJOR)
    ctx.synchronize()
    xd = x.double().cpu().numpy()
    for pay, y in zip(pays, ys):
        want = xd @ oracle.decompress(pay).astype(np.float64).T
        # fp32 sums of `cols` products, then of the codes: below sqrt(cols) * 2^-24
        assert np.linalg.norm(y.double().cpu().numpy() - want) <= 4e-6 * np.linalg.norm(want)


def test_a_group_whose_codes_leave_no_room_for_every_slice(ctx):
    """Three members of 28000 rows with 192 codes each: 225 KB of activations and codes a CTA, so that the
    slices of 780 atoms fit one at a time only."""
    rows, cols, atoms, slots = 28000, 1024, 780, 192
    pays = [synth.hsdr_payload(rows, cols, n_atoms=atoms, k=64, seed=i) for i in range(3)]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    x = np.random.default_rng(0).normal(0, 1, cols).astype(np.float32)
    xd, ys = torch.from_numpy(x).cuda(), [torch.full((rows,), float("nan"), device="cuda") for _ in pays]
    torch.cuda.synchronize()
    cs.Segment.matmul_group_device(segs, xd.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, 1, [y.data_ptr() for y in ys], cs.TOKEN_MAJOR)
    ctx.synchronize()
    for p, y in zip(pays, ys):
        at = 36 + 4 * 3
        dx = np.frombuffer(p, np.float32, atoms * cols, at).reshape(atoms, cols).astype(np.float64) @ x
        codes = np.frombuffer(p, np.uint16, rows * slots, at + 4 * atoms * cols).reshape(rows, slots)
        want = (dx[codes & 0x7FFF] * np.where(codes >> 15, -1.0, 1.0) * np.repeat([1.0, 0.5, 0.25], 64)).sum(axis=1)
        # fp32 sums of 1024 products, then of 192 codes
        assert np.linalg.norm(y.double().cpu().numpy() - want) <= 4e-6 * np.linalg.norm(want)

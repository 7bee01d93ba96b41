"""Whole-matrix reconstruction at the edges of its slices and tiles, bit-exact against the oracle."""
import struct

import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,tr,tc,atoms,k", [
    (300, 64, 1, 64, 128, 8),       # one slice exactly
    (301, 65, 1, 65, 100, 5),       # a slice and one element, odd stream
    (67, 4099, 1, 4099, 16, 3),     # odd width
    (128, 128, 32, 32, 16, 4),      # few tiles, aligned
    (131, 259, 16, 16, 24, 8),      # both strips, 128-bit stores refused
    (132, 260, 16, 16, 24, 5),      # both strips, 128-bit stores taken
    (96, 99, 4, 9, 40, 7),          # slice wider than the tile, rows of a tile not in fours
    (640, 96, 1, 96, 1000, 8),      # 32 elements a slice
    (20, 40, 4, 4, 8, 1),           # tiles below a slice: element-wise kernel
])
def test_reconstruction_is_bit_exact(ctx, oracle, rows, cols, tr, tc, atoms, k):
    pay = synth.hsdr_payload(rows, cols, tile_rows=tr, tile_cols=tc, n_atoms=atoms, k=k, seed=rows + cols)
    want = oracle.decompress(pay)
    seg = cs.Segment.from_payload(pay, ctx)
    got = torch.full((rows, cols), float("nan"), device="cuda")
    torch.cuda.synchronize()
    seg.decompress_device(got.data_ptr())
    ctx.synchronize()
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_tiles_that_span_more_than_32_bits(ctx):
    """4096-row tiles of a matrix 1049600 wide (17 GB): the last row of a tile lies past 2^32 elements."""
    rows, n_ct, tc, atoms = 4096, 262400, 4, 8
    rng = np.random.default_rng(0)
    d = rng.standard_normal((atoms, rows * tc), dtype=np.float32)
    codes = (rng.integers(0, atoms, n_ct) | rng.integers(0, 2, n_ct) << 15).astype(np.uint16)
    head = struct.pack("<4sIIIIHHHBBfI", b"HSDR", 2, rows, n_ct * tc, n_ct, rows, tc, atoms, 1, 1, 1.0, 0)
    seg = cs.Segment.from_payload(head + np.ones(1, np.float32).tobytes() + d.tobytes() + codes.tobytes(), ctx)
    got = torch.full((rows, n_ct, tc), float("nan"), device="cuda")
    torch.cuda.synchronize()
    seg.decompress_device(got.data_ptr())
    ctx.synchronize()
    c = torch.from_numpy(codes.astype(np.int64)).cuda()
    sign = (1.0 - 2.0 * (c >> 15)).float()[:, None]
    dt = torch.from_numpy(d).cuda().view(atoms, rows, tc)
    for r in (0, 1, 2047, 4094, 4095):
        assert torch.equal(got[r], dt[c & 0x7FFF, r] * sign)
    seg.close()

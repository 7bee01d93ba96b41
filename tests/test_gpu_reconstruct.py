"""Whole-matrix reconstruction at the edges of its slices and tiles, bit-exact against the oracle."""
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

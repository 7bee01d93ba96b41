"""More tokens, or tiles to encode, than a launch has token tiles in its grid's second dimension
(65535 of 64)."""
import struct

import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu

MOST = 65535 * 64


@pytest.mark.parametrize("rows,cols,tile", [(2, 3, 0), (3, 5, 2)])     # odd row tiles; ragged 2-D tiles
def test_products(ctx, oracle, rows, cols, tile):
    m = MOST + 65
    pay = synth.hsdr_payload(rows, cols, tile_rows=tile or 1, tile_cols=tile or cols, n_atoms=2, k=2, seed=1)
    seg = cs.Segment.from_payload(pay, ctx)
    x = torch.randn(m, cols, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    y = torch.full((m, rows), float("nan"), device="cuda")
    torch.cuda.synchronize()
    seg.matmul_device(x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, y.data_ptr(), cs.TOKEN_MAJOR)
    ctx.synchronize()
    want = x.double() @ torch.from_numpy(oracle.decompress(pay)).double().cuda().T
    # fp32 sums of at most five products
    assert (y.double() - want).norm() <= 1e-6 * want.norm() and (y[MOST:].double() - want[MOST:]).norm() <= 1e-6 * want[MOST:].norm()


def test_encoder(ctx):
    """2 x 2 tiles: every tile's one code names an atom of the largest projection."""
    w = np.random.default_rng(3).normal(0, 0.02, (4096, 4104)).astype(np.float32)
    pay = cs.HierarchicalSDRStrategy(ctx).compress(w, tile_rows=2, tile_cols=2, n_atoms=4, n_stages=1, k=1)
    n = 2048 * 2052
    assert n > MOST and struct.unpack_from("<I", pay, 16)[0] == n
    atoms = np.frombuffer(pay, np.float32, 16, 40).reshape(4, 4).astype(np.float64)
    codes = np.frombuffer(pay, np.uint16, n, 40 + 64)
    tiles = w.reshape(2048, 2, 2052, 2).transpose(0, 2, 1, 3).reshape(n, 4).astype(np.float64)
    dots = tiles @ atoms.T
    took = dots[np.arange(n), codes & 0x7FFF]
    off = 1e-6 * np.abs(tiles).max() * np.abs(atoms).max()        # fp32 projections of four products
    assert (np.abs(took) >= np.abs(dots).max(axis=1) - off).all()
    assert ((took < 0) == (codes >> 15 == 1))[np.abs(took) > off].all()

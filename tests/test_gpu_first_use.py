"""The first product with a weight, which builds planes of its dictionary, coefficient entries or the
rebuilt weight in front of kernels that read them ahead of their dependency wait, gives the bits of
the second; on the stream that built and on another."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,tile,m", [
    (640, 2048, 0, 8),          # planes, one token tile
    (2048, 1024, 0, 200),       # planes and entries
    (512, 2048, 128, 2),        # planes of a tile dictionary
    (512, 2048, 128, 32),       # planes of the rebuilt weight
    (700, 2100, 64, 24),        # the rebuilt weight itself
    (600, 2048, -1, 2),         # stage blocks: a list of one product
])
def test_first_is_second(rows, cols, tile, m):
    listed, tile = tile < 0, max(tile, 0)
    ctx, other = cs.Context(0), cs.Context(0)
    x = torch.randn(m, cols, generator=torch.Generator(device="cuda").manual_seed(m), device="cuda")
    y = [torch.full((m, rows), float("nan"), device="cuda") for _ in range(3)]
    pays = [synth.hsdr_payload(rows, cols, tile_rows=tile or 1, tile_cols=tile or cols, n_atoms=512, k=8, seed=i) for i in range(4)]

    def call(c, seg, out):
        if listed:
            task = (cs._lib.MatmulTask * 1)(cs._lib.MatmulTask(seg._h, x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, out.data_ptr(), cs.TOKEN_MAJOR, None, -1))
            cs._check(c._lib.csdr_matmul_queue_device_async(c._h, task, 1))
            return
        cs._check(c._lib.csdr_matmul_device_async(c._h, seg._h, x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, out.data_ptr(), cs.TOKEN_MAJOR, None))

    for i in range(12):
        seg = cs.Segment.from_payload(pays[i % 4], ctx)
        torch.cuda.synchronize()
        call(ctx, seg, y[0])
        if listed:
            ctx.synchronize()               # the list kernel wants the whole GPU for itself
        call(other, seg, y[1])              # behind the build, on a stream of its own
        if listed:
            other.synchronize()
        call(ctx, seg, y[2])
        ctx.synchronize()
        other.synchronize()
        assert torch.equal(y[0], y[2]) and torch.equal(y[1], y[2]) and torch.isfinite(y[2]).all()
        seg.close()
    ctx.close()
    other.close()

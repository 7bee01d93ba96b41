"""Products whose rebuilt weight has no room, by the context's budget or the device's, take the form
that needs none."""
import struct

import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,tile,m,bound", [
    (200, 300, 32, 40, 4e-6),        # edge strips: CUDA cores, fp32
    (300, 256, 32, 20, 2e-5),        # tile products on the tensor cores: two bf16 pieces of every operand
    (100, 102, 6, 3, 4e-6),          # rebuilt in scratch
])
def test_within_the_budget(oracle, monkeypatch, rows, cols, tile, m, bound):
    pay = synth.hsdr_payload(rows, cols, tile_rows=tile, tile_cols=tile, n_atoms=32, k=4, seed=rows)
    x = torch.from_numpy(np.random.default_rng(m).normal(0, 1, (m, cols)).astype(np.float32)).cuda()
    want = x.double().cpu().numpy() @ oracle.decompress(pay).astype(np.float64).T
    for megabytes in ("0", "1"):
        monkeypatch.setenv("CSDR_KEEP_MB", megabytes)
        ctx = cs.Context(0)
        segs = [cs.Segment.from_payload(pay, ctx) for _ in range(8)]
        y = torch.full((m, rows), float("nan"), device="cuda")
        torch.cuda.synchronize()
        for seg in segs:                 # the megabyte holds the first few: the rest go without
            for _ in range(2):
                y.fill_(float("nan"))
                torch.cuda.synchronize()
                seg.matmul_device(x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, y.data_ptr(), cs.TOKEN_MAJOR)
                ctx.synchronize()
                assert np.linalg.norm(y.double().cpu().numpy() - want) <= bound * np.linalg.norm(want)
        for seg in segs:
            seg.close()
        ctx.close()


def test_a_weight_larger_than_the_device(ctx):
    """220096 x 220032 in 64 x 128 tiles: 13 MB of codes, 194 GB as fp32."""
    n_rt, n_ct, tr, tc, atoms, m = 3439, 1719, 64, 128, 16, 16
    rng = np.random.default_rng(0)
    d = rng.standard_normal((atoms, tr * tc), dtype=np.float32)
    codes = (rng.integers(0, atoms, n_rt * n_ct) | rng.integers(0, 2, n_rt * n_ct) << 15).astype(np.uint16)
    head = struct.pack("<4sIIIIHHHBBfI", b"HSDR", 2, n_rt * tr, n_ct * tc, n_rt * n_ct, tr, tc, atoms, 1, 1, 1.0, 0)
    seg = cs.Segment.from_payload(head + np.ones(1, np.float32).tobytes() + d.tobytes() + codes.tobytes(), ctx)
    x = torch.randn(m, n_ct * tc, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    y = torch.full((m, n_rt * tr), float("nan"), device="cuda")
    torch.cuda.synchronize()
    seg.matmul_device(x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, m, y.data_ptr(), cs.TOKEN_MAJOR)
    ctx.synchronize()
    c = torch.from_numpy(codes.astype(np.int32)).cuda().view(n_rt, n_ct)
    sign = 1.0 - 2.0 * (c >> 15).double()
    dt, xt = torch.from_numpy(d).double().cuda().view(atoms, tr, tc), x.double().view(m, n_ct, tc)
    want = torch.zeros(n_rt, m * tr, dtype=torch.float64, device="cuda")
    for a in range(atoms):
        want += (sign * ((c & 0x7FFF) == a)) @ torch.einsum("mct,jt->cmj", xt, dt[a]).reshape(n_ct, m * tr)
    want = want.view(n_rt, m, tr).permute(1, 0, 2).reshape(m, n_rt * tr)
    assert (y.double() - want).norm() <= 2e-5 * want.norm()      # two bf16 pieces of every operand
    seg.close()

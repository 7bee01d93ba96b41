"""A call that is captured before what it would build on first use exists takes the form that needs
nothing built, and gives the same product when replayed."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,tile,warm,m", [
    (700, 512, 0, 64, 300),      # planes built by a smaller batch; the gather's entries are not
    (1500, 1000, 128, 0, 2),     # ragged tiles: no rebuilt weight yet
])
def test_first_use_under_capture(oracle, monkeypatch, rows, cols, tile, warm, m):
    def payload(r, atoms, **kw):
        return synth.hsdr_payload(r, cols, tile_rows=tile or 1, tile_cols=tile or cols, n_atoms=atoms, k=8, seed=r, **kw)

    st = torch.cuda.Stream()
    ctx = cs.Context(0, st.cuda_stream)
    monkeypatch.setenv("CSDR_GATHER_MMA", "0")
    monkeypatch.setenv("CSDR_CACHE_2D", "0")
    plain = cs.Context(0, st.cuda_stream)              # never builds what the captured call would
    pay = payload(rows, 128)
    seg = cs.Segment.from_payload(pay, ctx)
    # another segment that takes the fallback form anyway, so that the scratch has grown: stage scales
    # bf16 does not hold, or too many rows for the dense product to pay
    other = cs.Segment.from_payload(payload(40000, 128) if tile else payload(64, 512, decay=0.7), ctx)
    x = torch.from_numpy(np.random.default_rng(m).normal(0, 1, (m, cols)).astype(np.float32)).cuda()
    y, z = torch.zeros(m, rows, device="cuda"), torch.zeros(m, other.rows, device="cuda")
    torch.cuda.synchronize()

    def call(s, n, out):
        s.matmul_device(x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, n, out.data_ptr(), cs.TOKEN_MAJOR)

    if warm:
        call(seg, warm, y)
    call(other, m, z)
    ctx.synchronize()
    y.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        call(seg, m, y)
    g.replay()
    torch.cuda.synchronize()
    want = x.double().cpu().numpy() @ oracle.decompress(pay).astype(np.float64).T
    # two bf16 pieces of every operand in the first case, fp32 in the second
    assert np.linalg.norm(y.double().cpu().numpy() - want) <= 2e-5 * np.linalg.norm(want)
    # the form that needs nothing built, to the bit; the call outside the capture takes the other one
    bare = cs.Segment.from_payload(pay, plain)
    y_plain, y_later = torch.zeros_like(y), torch.zeros_like(y)
    call(bare, m, y_plain)
    call(seg, m, y_later)
    plain.synchronize()
    ctx.synchronize()
    assert torch.equal(y, y_plain) and not torch.equal(y, y_later)
    bare.close()
    del g
    seg.close()
    other.close()

"""The encoder's workspaces: not those a captured product writes, and not kept past 256 MB each."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cache", ["1", "0"])     # tile products on the tensor cores; a weight rebuilt in scratch
def test_a_captured_product_outlives_an_encode(oracle, monkeypatch, cache):
    monkeypatch.setenv("CSDR_CACHE_2D", cache)
    monkeypatch.setenv("CSDR_TILE_TC", cache)
    st = torch.cuda.Stream()
    ctx = cs.Context(0, st.cuda_stream)
    cols = 512 if cache == "1" else 510               # 510: tiles that are no multiple of four columns
    pay = synth.hsdr_payload(256, cols, tile_rows=32, tile_cols=32 if cache == "1" else 30, n_atoms=16, k=4, seed=1)
    seg = cs.Segment.from_payload(pay, ctx)
    x = torch.randn(2, cols, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    y = torch.empty(2, 256, device="cuda")
    torch.cuda.synchronize()

    def call():
        seg.matmul_device(x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, 2, y.data_ptr(), cs.TOKEN_MAJOR)

    call()
    ctx.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        call()
    w = np.random.default_rng(0).normal(0, 0.02, (1024, 1024)).astype(np.float32)
    cs.HierarchicalSDRStrategy(ctx).compress(w, tile_rows=32, tile_cols=32, n_atoms=128, k=4)
    hold = [torch.zeros(1 << 20, device="cuda") for _ in range(8)]     # whatever memory had been given back
    y.fill_(float("nan"))
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    want = x.double().cpu().numpy() @ oracle.decompress(pay).astype(np.float64).T
    assert np.linalg.norm(y.double().cpu().numpy() - want) <= 2e-5 * np.linalg.norm(want)     # two bf16 pieces of every operand
    assert not any(h.any() for h in hold)
    del g
    seg.close()


def test_large_workspaces_are_given_back():
    ctx = cs.Context(0)
    enc = cs.HierarchicalSDRStrategy(ctx)
    rng = np.random.default_rng(1)
    tiles, atoms = rng.normal(0, 1, (600_000, 8)).astype(np.float32), rng.normal(0, 1, (128, 8)).astype(np.float32)
    enc.encode_codes(tiles[:1000], atoms, np.ones(1, np.float32), 1)
    before = torch.cuda.mem_get_info()[0]
    enc.encode_codes(tiles, atoms, np.ones(1, np.float32), 1)          # 307 MB of projections
    assert torch.cuda.mem_get_info()[0] >= before - (128 << 20)
    enc.compress_shared([tiles.reshape(1200, 4000)], tile_rows=2, tile_cols=4, n_atoms=128, n_stages=1, k=1)
    assert torch.cuda.mem_get_info()[0] >= before - (128 << 20)
    ctx.close()

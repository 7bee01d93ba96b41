"""The gather as a matrix product on the tensor cores against the lookups in shared memory (the same
projection in front of both) and against 64-bit products: row tiles and token slices around their
edges, dictionaries of two to eight blocks, blocks with more entries than a thread keeps, atoms named
twice by a row, bias, both layouts; stage scales it does not take stay with the lookups."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


def run(monkeypatch, on, pays, x, dtype, token, bias):
    monkeypatch.setenv("CSDR_GATHER_MMA", on)
    monkeypatch.setenv("CSDR_GATHER_MMA_MIN", "17")
    ctx = cs.Context(0)
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    t = torch.from_numpy(x).cuda()
    t = t.bfloat16() if dtype == "bf16" else t
    m, layout = x.shape[0], cs.TOKEN_MAJOR if token else cs.FEATURE_MAJOR
    xin = t.contiguous() if token else t.t().contiguous()
    ys = [torch.full((m, s.rows) if token else (s.rows, m), float("nan"), device="cuda") for s in segs]
    bd = torch.from_numpy(bias).cuda() if bias is not None else None
    code = cs.DTYPE_BF16 if dtype == "bf16" else cs.DTYPE_F32
    torch.cuda.synchronize()
    for _ in range(2):
        if len(segs) > 1:
            cs.Segment.matmul_group_device(segs, xin.data_ptr(), code, layout, m, [y.data_ptr() for y in ys], layout)
        else:
            segs[0].matmul_device(xin.data_ptr(), code, layout, m, ys[0].data_ptr(), layout, bd.data_ptr() if bd is not None else 0)
    ctx.synchronize()
    out = [(y if token else y.t()).double().cpu().numpy() for y in ys]
    xd = t.double().cpu().numpy()
    for s in segs:
        s.close()
    ctx.close()
    return out, xd


def check(oracle, monkeypatch, pays, x, dtype, token, bias=None):
    got, xd = run(monkeypatch, "1", pays, x, dtype, token, bias)
    look, _ = run(monkeypatch, "0", pays, x, dtype, token, bias)
    for g, l, pay in zip(got, look, pays):
        want = xd @ oracle.decompress(pay).astype(np.float64).T + (0 if bias is None else bias)
        # the same 24-bit projection, at most 64 exact terms in fp32: 64 * 2^-24 at the very most
        assert np.linalg.norm(g - l) <= 2e-6 * np.linalg.norm(l)
        # two 8-bit pieces of every operand in the projection: 2^-17
        assert np.linalg.norm(g - want) <= 2e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("dtype,token", [("f32", False), ("f32", True), ("bf16", False), ("bf16", True)])
@pytest.mark.parametrize("rows,atoms,k,m", [
    (1, 128, 8, 64),         # one row, one slice
    (127, 128, 1, 65),       # a slice and a token
    (128, 256, 8, 128),
    (129, 512, 8, 97),       # a row tile and a row; tokens not in fours
    (1500, 384, 5, 40),      # part of a slice, six blocks
    (3000, 512, 21, 200),    # 63 codes a row: more entries a block than a thread keeps
])
def test_gather_products(oracle, monkeypatch, rows, atoms, k, m, dtype, token):
    pay = synth.hsdr_payload(rows, 192, n_atoms=atoms, k=k, seed=rows + atoms)
    rng = np.random.default_rng(m)
    x, bias = rng.normal(0, 1, (m, 192)).astype(np.float32), rng.normal(0, 1, rows).astype(np.float32)
    check(oracle, monkeypatch, [pay], x, dtype, token, bias)


def test_gather_products_of_a_group(oracle, monkeypatch):
    pays = [synth.hsdr_payload(r, 128, n_atoms=a, k=8, seed=r) for r, a in ((300, 128), (130, 512), (700, 256))]
    x = np.random.default_rng(0).normal(0, 1, (150, 128)).astype(np.float32)
    check(oracle, monkeypatch, pays, x, "bf16", True)


@pytest.mark.parametrize("decay", [0.7, 0.0625])   # not exact in bf16; exact, but the sums are not
def test_other_stage_scales(oracle, monkeypatch, decay):
    pay = synth.hsdr_payload(200, 128, n_atoms=128, k=8, decay=decay, seed=4)
    x = np.random.default_rng(1).normal(0, 1, (70, 128)).astype(np.float32)
    check(oracle, monkeypatch, [pay], x, "f32", True)

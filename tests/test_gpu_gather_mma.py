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
    counts = [ctx.launch_count]
    for _ in range(2):
        if len(segs) > 1:
            cs.Segment.matmul_group_device(segs, xin.data_ptr(), code, layout, m, [y.data_ptr() for y in ys], layout)
        else:
            segs[0].matmul_device(xin.data_ptr(), code, layout, m, ys[0].data_ptr(), layout, bd.data_ptr() if bd is not None else 0)
        counts.append(ctx.launch_count)
    ctx.synchronize()
    built = counts[1] - counts[0] - (counts[2] - counts[1])        # launches only the first call had
    out = [(y if token else y.t()).double().cpu().numpy() for y in ys]
    xd = t.double().cpu().numpy()
    for s in segs:
        s.close()
    ctx.close()
    return out, xd, built


def check(oracle, monkeypatch, pays, x, dtype, token, bias=None, taken=True):
    """taken: the products go to the tensor cores (their entries are built, a launch a segment, and their
    sums have another order than the lookups'); else both runs are the lookups'."""
    got, xd, built = run(monkeypatch, "1", pays, x, dtype, token, bias)
    look, _, planes = run(monkeypatch, "0", pays, x, dtype, token, bias)
    assert built - planes == (len(pays) if taken else 0)
    assert taken or all(np.array_equal(g, l) for g, l in zip(got, look))
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
    check(oracle, monkeypatch, [pay], x, "f32", True, taken=False)


@pytest.mark.parametrize("token", [False, True])
def test_values_that_are_not_finite_stay_in_the_rows_that_name_them(monkeypatch, token):
    """A bad atom, a projection past fp32, one past what bf16 rounds to, a bad token: the same infinities
    and NaN as the lookups, and none elsewhere."""
    rows, cols, atoms, m, big = 300, 192, 512, 150, 11
    pay = bytearray(synth.hsdr_payload(rows, cols, n_atoms=atoms, k=8, seed=9))
    d = np.frombuffer(pay, np.float32, atoms * cols, 36 + 4 * 3).reshape(atoms, cols)   # behind the header and the stage scales
    d[7, 100] = np.inf
    d[20:, :big] = 0
    d[20, :big - 1] = 2.0 ** np.arange(127, 127 - big + 1, -1)      # their sum: 2^128 (1 - 2^-10)
    d[21, 0] = 2.0 ** 127
    x = np.random.default_rng(2).normal(0, 1, (m, cols)).astype(np.float32)
    x[:, :big] = 0
    x[70, :big] = 1                                    # finite in fp32, past bf16's rounding
    x[71, 0] = 64                                      # past fp32
    x[140, 50] = np.nan
    got, _, _ = run(monkeypatch, "1", [bytes(pay)], x, "f32", token, None)
    look, _, _ = run(monkeypatch, "0", [bytes(pay)], x, "f32", token, None)
    codes = np.frombuffer(bytes(pay), np.uint16, rows * 24, 36 + 4 * 3 + 4 * atoms * cols).reshape(rows, 24) & 0x7FFF
    clean = ~np.isin(codes, (7, 20, 21)).any(axis=1)
    assert 100 < clean.sum() < rows
    fine = np.ones(m, bool)
    fine[140] = False
    assert np.isfinite(look[0][np.ix_(fine, clean)]).all() and np.isnan(look[0][140]).all()
    assert not np.isfinite(look[0][np.ix_(fine, (codes == 7).any(axis=1))]).any()
    assert np.isfinite(look[0][70, (codes[:, 16:] == 20).any(axis=1) & ~(codes[:, :16] == 20).any(axis=1) & ~np.isin(codes, (7, 21)).any(axis=1)]).all()
    # the same 24-bit projection, 24 exact terms in fp32
    np.testing.assert_allclose(got[0], look[0], rtol=1e-4, atol=1e-6 * np.abs(x[fine]).max(), equal_nan=True)

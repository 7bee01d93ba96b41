"""Lists the list kernel does not take give what their tasks give one after the other, also where a
task reads or overwrites what an earlier one wrote or read without naming it; groups likewise."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu

FP32 = 4e-6     # sums of 45 products of 24-bit operands in fp32, then of the codes


def dense(pay, oracle):
    return oracle.decompress(pay).astype(np.float64)


def check(got, want):
    assert np.linalg.norm(got.double().cpu().numpy() - want) <= FP32 * np.linalg.norm(want)


@pytest.mark.parametrize("n,first", [(5, 45), (40, 45), (40, 31)])     # 40: past a group of 32 and a launch's members
def test_a_chain_that_names_nothing(ctx, oracle, n, first):
    """Task i reads task i - 1's result; the first product may have another width."""
    pays = [synth.hsdr_payload(45, first if i == 0 else 45, n_atoms=20, k=4, seed=i, weight_std=0.15) for i in range(n)]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    # a gain near one, so that forty products in a row stay in range
    x = torch.from_numpy(np.random.default_rng(n).normal(0, 1, (2, first)).astype(np.float32)).cuda()
    ys = [torch.full((2, 45), float("nan"), device="cuda") for _ in range(n)]
    torch.cuda.synchronize()
    cs.Segment.matmul_queue_device([(s, (x if i == 0 else ys[i - 1]).data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, 2, ys[i].data_ptr(), cs.TOKEN_MAJOR)
                                    for i, s in enumerate(segs)])
    ctx.synchronize()
    for i, p in enumerate(pays):                       # each link from what the one before it gave
        check(ys[i], (x if i == 0 else ys[i - 1]).double().cpu().numpy() @ dense(p, oracle).T)


def test_results_that_lie_on_earlier_operands(ctx, oracle):
    pays = [synth.hsdr_payload(45, 45, n_atoms=20, k=4, seed=i) for i in range(6)]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    ws = [dense(p, oracle) for p in pays]
    rng = np.random.default_rng(1)
    a, b = (torch.from_numpy(rng.normal(0, 1, (2, 45)).astype(np.float32)).cuda() for _ in range(2))
    bias = torch.from_numpy(rng.normal(0, 1, 45).astype(np.float32)).cuda()
    ad, bd, biasd = a.double().cpu().numpy(), b.double().cpu().numpy(), bias.double().cpu().numpy()
    y = [torch.full((2, 45), float("nan"), device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    f = (cs.DTYPE_F32, cs.TOKEN_MAJOR, 2)
    cs.Segment.matmul_queue_device([
        (segs[0], a.data_ptr(), *f, y[0].data_ptr(), cs.TOKEN_MAJOR, bias.data_ptr()),
        (segs[1], a.data_ptr(), *f, y[1].data_ptr(), cs.TOKEN_MAJOR),
        (segs[2], b.data_ptr(), *f, y[1].data_ptr(), cs.TOKEN_MAJOR),          # the same result again: the later one stays
        (segs[3], b.data_ptr(), *f, a.data_ptr(), cs.TOKEN_MAJOR),             # over activations read before
        (segs[4], a.data_ptr(), *f, y[2].data_ptr(), cs.TOKEN_MAJOR),          # which are now that result
        (segs[5], b.data_ptr(), *f, y[3].data_ptr(), cs.TOKEN_MAJOR, y[1].data_ptr()),   # a bias that is a result
    ])
    ctx.synchronize()
    check(y[0], ad @ ws[0].T + biasd)
    check(y[1], bd @ ws[2].T)
    check(a, bd @ ws[3].T)
    check(y[2], a.double().cpu().numpy() @ ws[4].T)
    check(y[3], bd @ ws[5].T + y[1].double().cpu().numpy()[0])


def test_a_group_that_overwrites_its_activations(ctx, oracle):
    pays = [synth.hsdr_payload(45, 45, n_atoms=20, k=4, seed=10 + i) for i in range(2)]
    segs = [cs.Segment.from_payload(p, ctx) for p in pays]
    x = torch.from_numpy(np.random.default_rng(2).normal(0, 1, (2, 45)).astype(np.float32)).cuda()
    xd, y = x.double().cpu().numpy(), torch.full((2, 45), float("nan"), device="cuda")
    torch.cuda.synchronize()
    cs.Segment.matmul_group_device(segs, x.data_ptr(), cs.DTYPE_F32, cs.TOKEN_MAJOR, 2, [x.data_ptr(), y.data_ptr()], cs.TOKEN_MAJOR)
    ctx.synchronize()
    check(x, xd @ dense(pays[0], oracle).T)
    check(y, x.double().cpu().numpy() @ dense(pays[1], oracle).T)

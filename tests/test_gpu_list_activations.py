"""Lists of products whose activations the list kernel cannot copy in bulk: two to four feature-major
tokens, bf16, rows off 16-byte boundaries - staged as fp32 rows before the list, alone and mixed with
rows that need nothing, one activation shared by several members."""
import numpy as np
import pytest
import torch

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [4, 1028, 2048])     # below a slab, one float4 past one, two
@pytest.mark.parametrize("m", [1, 2, 3, 4])
def test_list_activations(ctx, oracle, cols, m):
    rng = np.random.default_rng(cols + m)
    forms = [(cs.DTYPE_F32, cs.FEATURE_MAJOR, 0), (cs.DTYPE_BF16, cs.FEATURE_MAJOR, 0), (cs.DTYPE_F32, cs.TOKEN_MAJOR, 0),
             (cs.DTYPE_BF16, cs.TOKEN_MAJOR, 0), (cs.DTYPE_F32, cs.TOKEN_MAJOR, 1), (cs.DTYPE_BF16, cs.FEATURE_MAJOR, 0)]
    tasks, keep, ys, xs = [], [], [], []
    for i, (dtype, layout, shift) in enumerate(forms):
        pay = synth.hsdr_payload(67 + i, cols, n_atoms=40 + 8 * i, k=8, seed=i)
        seg = cs.Segment.from_payload(pay, ctx)
        if i == 5:                                     # the second member's activation again
            x, view = xs[1], tasks[1][1]
        else:
            x = torch.from_numpy(rng.normal(0, 1, (m, cols)).astype(np.float32)).cuda()
            x = x.bfloat16() if dtype == cs.DTYPE_BF16 else x
            mem = x if layout == cs.TOKEN_MAJOR else x.t().contiguous()
            room = torch.empty(mem.numel() + shift, dtype=mem.dtype, device="cuda")
            room[shift:] = mem.reshape(-1)
            keep.append(room)
            view = room.data_ptr() + shift * room.element_size()
        y = torch.full((seg.rows, m), float("nan"), device="cuda")
        xs.append(x)
        ys.append((y, oracle.decompress(pay)))
        tasks.append((seg, view, dtype, layout, m, y.data_ptr(), cs.FEATURE_MAJOR))
    torch.cuda.synchronize()
    prepared = cs.Segment.matmul_queue_device(tasks)
    cs.Segment.matmul_queue_device(None, prepared)
    ctx.synchronize()
    for x, (y, w) in zip(xs, ys):
        want = w.astype(np.float64) @ x.double().cpu().numpy().T
        # fp32 sums of `cols` products: below sqrt(cols) * 2^-24
        assert np.linalg.norm(y.double().cpu().numpy() - want) <= 3e-6 * np.linalg.norm(want)

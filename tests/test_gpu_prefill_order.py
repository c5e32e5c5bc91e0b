"""The order in which a launch takes its query tiles (by tiles, by pairs because of the first sequence's past, by pairs
because of the launch's size) changes no bit of a sequence's output."""
from __future__ import annotations

import pytest
import torch

from compactor_vllm.attention.sparse_varlen_kernel import causal_sparse_varlen_with_cache

from helpers import fused_qkv, make_paged

pytestmark = pytest.mark.gpu
DEV = "cuda"
HQ, HKV, PS, D = 32, 8, 128, 128


def _run(seqs, new, past, pools):
    """Outputs per sequence of one call over the sequences `seqs`, in that order."""
    q, k, v, cu, kc, vc, pt, bm = pools
    rows = torch.cat([torch.arange(int(cu[i]), int(cu[i + 1])) for i in seqs]).to(DEV)
    cu_call = torch.tensor([0] + [new[i] for i in seqs]).cumsum(0).to(torch.int32)
    lens = torch.tensor([[past[i]] * HKV for i in seqs], dtype=torch.int32, device=DEV)
    out = causal_sparse_varlen_with_cache(q[rows], k[rows], v[rows], kc, vc, lens, pt, bm[list(seqs)].contiguous(),
                                          cu_call.to(DEV), max(new[i] for i in seqs), int(lens.max()), HKV, PS, None)
    torch.cuda.synchronize()
    return dict(zip(seqs, out.split([new[i] for i in seqs])))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("new,past,calls", [
    # whole tiles of 128: a ragged tail's tile also holds rows of whatever sequence comes next, and the rows of a warp
    # move their softmax reference point together (ragged tails against the oracle: test_gpu_prefill.py)
    ([640, 256, 128], [0, 600, 1], [(0, 1, 2), (1, 0, 2), (2, 1, 0)]),          # the first past: 0, 600, 1
    ([384] * 40, [0, 70] * 20, [tuple(range(40)), tuple(range(20)), tuple(range(20, 40))]),   # 1920 CTAs; 960
])
def test_order_changes_nothing(dtype, new, past, calls):
    kc, vc, pt, bm = make_paged(len(new), HKV, D, PS, [[n] * HKV for n in past], dtype, DEV, seed=3, poison=True)
    cu = torch.tensor([0] + new).cumsum(0)
    q, k, v = fused_qkv(int(cu[-1]), HQ, HKV, D, dtype, DEV, seed=4)
    pools = (q, k, v, cu, kc, vc, pt, bm)
    want = _run(calls[0], new, past, pools)
    assert all(torch.isfinite(o).all() for o in want.values())
    for call in calls[1:]:
        for i, o in _run(call, new, past, pools).items():
            assert torch.equal(o, want[i]), i

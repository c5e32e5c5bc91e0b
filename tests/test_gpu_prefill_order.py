"""The order in which a launch takes its query tiles (by tiles, by pairs because of the pasts, by pairs because of the
launch's size) changes no bit of a sequence's output."""
from __future__ import annotations

import pytest
import torch

from compactor_vllm.attention.sparse_varlen_kernel import causal_sparse_varlen_with_cache

from helpers import fused_qkv, make_paged

pytestmark = pytest.mark.gpu
DEV = "cuda"
HQ, HKV, PS, D = 32, 8, 128, 128


def _run(seqs, new, past, pools, bound=None):
    """Outputs per sequence of one call over the sequences `seqs`, in that order; `bound`: what it is told of the pasts."""
    q, k, v, cu, kc, vc, pt, bm = pools
    rows = torch.cat([torch.arange(int(cu[i]), int(cu[i + 1])) for i in seqs]).to(DEV)
    cu_call = torch.tensor([0] + [new[i] for i in seqs]).cumsum(0).to(torch.int32)
    lens = torch.tensor([[past[i]] * HKV for i in seqs], dtype=torch.int32, device=DEV)
    out = causal_sparse_varlen_with_cache(q[rows], k[rows], v[rows], kc, vc, lens, pt, bm[list(seqs)].contiguous(),
                                          cu_call.to(DEV), max(new[i] for i in seqs), int(lens.max()) if bound is None else bound,
                                          HKV, PS, None)
    torch.cuda.synchronize()
    return dict(zip(seqs, out.split([new[i] for i in seqs])))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("new,past,calls", [
    # whole tiles of 128: a ragged tail's tile also holds rows of whatever sequence comes next, and the rows of a warp
    # move their softmax reference point together (ragged tails against the oracle: test_gpu_prefill.py)
    ([640, 256, 128], [0, 600, 1], [(0, 1, 2), (1, 0, 2), (2, 1, 0)]),          # by pairs for the pasts, in three batch orders
    ([1280, 640, 128], [0, 2600, 1], [(0, 1, 2), (2, 0), (2, 1, 0), (1, 2)]),   # by pairs for the pasts; by tiles; pairs; one wave
    ([1280, 640], [0, 100], [(0, 1), (0,), (1,)]),     # CTAs go on with other tiles; 160 CTAs, which don't; one wave
    ([1280, 640], [2600, 0], [(0, 1), (0,)]),          # the same by pairs
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


@pytest.mark.parametrize("bound", [0, 959, 961, 2 ** 40, -1])
def test_the_bound_of_the_pasts_only_orders(bound):
    """By tiles up to three quarters of the longest prompt (960), by pairs beyond; a bound that is wrong costs speed alone."""
    new, past = [1280, 384, 128], [500, 2600, 0]
    kc, vc, pt, bm = make_paged(3, HKV, D, PS, [[n] * HKV for n in past], torch.bfloat16, DEV, seed=5, poison=True)
    cu = torch.tensor([0] + new).cumsum(0)
    q, k, v = fused_qkv(int(cu[-1]), HQ, HKV, D, torch.bfloat16, DEV, seed=6)
    pools = (q, k, v, cu, kc, vc, pt, bm)
    want, got = _run((0, 1, 2), new, past, pools), _run((0, 1, 2), new, past, pools, bound)
    assert all(torch.equal(got[i], want[i]) and torch.isfinite(got[i]).all() for i in want)


def _order(past, tiles, pairs, seqs, tokens):
    """What the CTAs of a biased launch take, (tile, pair, sequence) each in launch order, and whether it looked at the pasts."""
    import ctypes
    from compactor_vllm import _native as N

    p = torch.tensor(past, dtype=torch.int32, device=DEV)
    out = torch.full((tiles * pairs * seqs, 3), -1, dtype=torch.int32, device=DEV)
    by_tile = ctypes.c_int()
    N.check(N.lib().cvllm_selftest_tile_order(N.ptr(p), p.numel(), tiles, pairs, seqs, tokens, 128, N.ptr(out),
                                              ctypes.byref(by_tile), N.stream(p.device)), "cvllm_selftest_tile_order")
    return [tuple(x) for x in out.tolist()], bool(by_tile.value)


def test_the_order_does_not_depend_on_which_sequence_is_first():
    """The same batch in another order of its sequences takes the same schedule; every CTA gets a tile of its own."""
    tiles, pairs, seqs = 16, 8, 5
    everything = {(t, p, b) for t in range(tiles) for p in range(pairs) for b in range(seqs)}
    for past in ([0, 8000, 8000, 8000, 8000], [0, 0, 0, 0, 4000], [1023] * 5, [1025] * 5):
        kinds = set()
        for turn in range(seqs):
            got, looked = _order(past[turn:] + past[:turn], tiles, pairs, seqs, tiles * 128 * seqs)
            assert looked and set(got) == everything
            kinds.add([t for t, _, _ in got] == sorted((t for t, _, _ in got), reverse=True))   # by tiles?
        assert kinds == {2 * sum(past) <= seqs * tiles * 128}, past


def test_tiles_past_the_end_of_short_sequences_do_not_count():
    """4000 + 2077 + 911 + 3301 tokens, 16 pairs: 2048 CTAs in the grid, at most (80 + 4) * 16 = 1344 with work."""
    n = 4000 + 2077 + 911 + 3301
    assert _order([0] * 4, 32, 16, 4, n)[1]
    assert not _order([0] * 4, 32, 16, 4, 32 * 128 * 4)[1]
    assert not _order([0], 9, 16, 1, 1100)[1]     # one wave

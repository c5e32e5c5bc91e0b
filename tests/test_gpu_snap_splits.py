"""Observation-window scores over the ways a call is cut into key splits: one tile per split, several, splits
beyond a short sequence, many (sequence, head) pairs with the fixed split; fewer rows than the tile has."""
from __future__ import annotations

import pytest
import torch

from compactor_vllm.compression.snapkv import query_aware_key_scores
from oracle import scoring as osc

from helpers import fused_qkv

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [
    ([33], 8, 8, 32),                          # one scored key
    ([32 + 128], 32, 8, 32),                   # exactly one tile of scored keys, the window in a split of its own
    ([18 * 128 + 31], 32, 8, 32),              # one tile per split, as many splits as there are CTAs
    ([2 * 18 * 128 + 129], 32, 8, 32),         # the first length that takes three tiles per split
    ([9000], 3, 1, 32),                        # 96 of 128 rows, one head: 71 tiles on 148 CTAs
    ([40, 6000, 32, 1, 129], 16, 4, 32),       # unequal sequences: more waves, empty splits
    ([1300, 700, 260, 64, 33, 2200, 90, 515, 300, 1025], 16, 8, 16),   # 80 pairs: the fixed split, 32 rows
    ([33, 500, 9000], 16, 2, 32),              # two row tiles, both full
    ([200, 3000], 8, 1, 17),                   # two row tiles, 8 rows in the second
    ([5000], 12, 2, 40),                       # 240 rows
    ([1300, 700, 260, 64, 33, 2200, 90, 515, 300, 1025] * 4, 16, 2, 32),   # 80 pairs of two row tiles: the fixed split
]


@pytest.mark.parametrize("lens,hq,hkv,w", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_splits_match_oracle(lens, hq, hkv, w, dtype):
    q, k, _ = fused_qkv(sum(lens), hq, hkv, 128, dtype, DEV, seed=sum(lens) + hq)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    for seg in (128, 32):
        out = query_aware_key_scores(q, k, cu.to(DEV), cu.to(DEV), w, pool_segment=seg).cpu()
        ref = osc.query_aware_key_scores(q.cpu(), k.cpu(), cu, cu, w, pool_segment=seg).float()
        assert torch.equal(torch.isinf(out), torch.isinf(ref))
        ok = torch.isfinite(ref)
        # both sides work in 32 bits from the same 16-bit inputs: a logit of size <= 16 differs by less than 2^-16,
        # 128 products of 2^-24 each, and its exponential by as much relative to itself, once in the
        # numerator and once in the row's sum
        assert ((out[ok] - ref[ok]).abs() <= 4 * 2**-16 * ref[ok].abs() + 1e-7).all()


@pytest.mark.parametrize("hq,hkv,w", [(32, 8, 32), (16, 2, 32), (4, 4, 1)])
def test_queries_packed_otherwise_than_keys(hq, hkv, w):
    """The query window ends where cu_seqlens_q says, in a packing with more tokens than the keys'."""
    lens = [300, 40, 1111]
    q, _, _ = fused_qkv(3 * sum(lens), hq, hkv, 128, torch.bfloat16, DEV, seed=1)
    _, k, _ = fused_qkv(sum(lens), hq, hkv, 128, torch.bfloat16, DEV, seed=2)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    out = query_aware_key_scores(q, k, (3 * cu).to(DEV), cu.to(DEV), w).cpu()
    tail = torch.cat([q[3 * e - n:3 * e] for e, n in zip(cu[1:].tolist(), lens)]).contiguous()
    assert torch.equal(out, query_aware_key_scores(tail, k, cu.to(DEV), cu.to(DEV), w).cpu())


@pytest.mark.parametrize("hq,hkv,w", [(32, 8, 32), (16, 2, 32), (4, 4, 1)])
def test_queries_past_the_end_count_as_zeros(hq, hkv, w):
    lens, short = [300, 40, 1111], 5
    q, k, _ = fused_qkv(sum(lens), hq, hkv, 128, torch.bfloat16, DEV, seed=7)
    q[-short:] = 0
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    assert torch.equal(query_aware_key_scores(q[:-short], k, cu, cu, w), query_aware_key_scores(q, k, cu, cu, w))


def test_no_window_scores_nothing():
    from compactor_vllm import _native as N

    q, k, _ = fused_qkv(300, 8, 2, 128, torch.float16, DEV, seed=3)
    cu, out = torch.tensor([0, 300], dtype=torch.int32, device=DEV), torch.full((300, 2), 7.0, device=DEV)
    ws = torch.empty(1 << 20, dtype=torch.uint8, device=DEV)
    N.check(N.lib().cvllm_snapkv_scores(q, k, q.stride(0), k.stride(0), cu, cu, 0, 1, 300, 8, 2, 128, 300, 0.1, 5, 64, out, 0, ws,
                                        ws.numel(), N.stream(out.device)), "snapkv")
    assert (out == 0).all()

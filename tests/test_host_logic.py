"""Host-side logic of the path against values produced by the REFERENCE's own functions
(oracle/gen_golden.py `splits` / `memory`): no GPU, no compute calls."""
import dataclasses

import pytest

from conftest import load_golden


def test_num_splits_heuristic_matches_reference():
    """attention/sparse_decode_kernel.py:168-192 over (b x kv-head blocks, context, SMs, split cap)."""
    from compactor_vllm.attention.sparse_decode_kernel import num_splits_heuristic

    table = load_golden("num_splits")["table"]
    assert table.shape[0] > 2000
    for blocks, seq, sms, cap, want in table.tolist():
        assert num_splits_heuristic(blocks, seq, sms, cap) == want, (blocks, seq, sms, cap)
    # the engine's capture-time call on this part: B=1, 8 kv heads, 32K context, 148 SMs
    assert num_splits_heuristic(8, 32768, 148, 64) >= 2


def test_kv_page_budget_matches_reference():
    """core/memory_manager.py:92-126 on scripted allocator readings (incl. the two RuntimeError exits)."""
    from compactor_vllm.core.memory_manager import MemorySnapshot, kv_page_budget

    g = load_golden("memory_budget")
    seen_error = seen_pages = 0
    for total, used, peak, cur, pct, layers, heads, hd, ps, esz, nb, nlp, want in g["pages"].tolist():
        snap = MemorySnapshot(total, total - used, peak, cur)
        kw = dict(num_layers=layers, heads=heads, head_dim=hd, page_size=ps, elem_size=esz, max_batches=nb,
                  logical_pages=nlp)
        if want < 0:
            with pytest.raises(RuntimeError):
                kv_page_budget(snap, pct / 100, **kw)
            seen_error += 1
        else:
            assert kv_page_budget(snap, pct / 100, **kw) == want
            seen_pages += 1
    assert seen_error > 0 and seen_pages > 0


def test_activation_token_budget_matches_reference():
    """core/memory_manager.py:128-161."""
    from compactor_vllm.core.memory_manager import MemorySnapshot, activation_token_budget

    rows = load_golden("memory_budget")["tokens"].tolist()
    assert rows
    for total, used, peak, cur, pct, heads, ps, pages, wt, before, after, want in rows:
        snap = MemorySnapshot(total, total - used, peak, cur)
        got = activation_token_budget(snap, pct / 100, warmup_tokens=wt, used_before=before, peak_after=after,
                                      num_pages=pages, page_size=ps, heads=heads)
        assert got == want


def test_context_records_are_dataclasses():
    """utils/context.py:10-40: `dataclasses.replace / asdict / fields` are legal on the reference's records."""
    from compactor_vllm.utils.context import CompressionContext, Context, get_context, reset_context, set_context

    names = [f.name for f in dataclasses.fields(Context)]
    # the reference's fields in the reference's order, then the ones mixed steps add
    assert names == ["is_prefill", "do_compression", "cu_seqlens_q", "cu_seqlens_k", "max_seqlen_q", "max_seqlen_k",
                     "batch_mapping", "max_bh_len", "compression_context", "STORE_STREAM", "key_split",
                     "attention_backend", "positions_i32", "token_slot", "seq_start"]
    assert [f.name for f in dataclasses.fields(CompressionContext)] == [
        "compression_method", "compression_chunk_size", "batch_tokens_to_retain", "max_tokens_to_retain",
        "context_lens", "PHI", "protected_first_tokens", "protected_last_tokens"]
    c = Context(True, True, max_bh_len=7)
    assert dataclasses.replace(c, max_bh_len=9).max_bh_len == 9 and c.max_bh_len == 7
    assert dataclasses.asdict(CompressionContext(context_lens=[3]))["context_lens"] == [3]
    with pytest.raises(TypeError):
        Context(no_such_field=1)
    set_context(is_prefill=True, max_seqlen_q=4)
    assert get_context().is_prefill and get_context().max_seqlen_q == 4
    reset_context()
    assert not get_context().is_prefill


def test_slot_map_reuses_and_releases():
    from compactor_vllm.core.memory_manager import SlotMap

    class FakeCache:
        def __init__(self):
            self.free, self.freed = [3, 2, 1], []

        def new_batch(self):
            return self.free.pop() if self.free else None

        def free_batch(self, slot):
            self.freed.append(slot)

    cache, slots = FakeCache(), SlotMap()
    assert [slots.acquire(cache, s) for s in (10, 11, 10, 12, 13)] == [1, 2, 1, 3, None]
    slots.release(cache, 11)
    assert cache.freed == [2] and 11 not in slots.by_seq


def test_shape_envelope_is_checked_at_construction():
    """D != 128 etc. are refused by name before any kernel is launched."""
    from types import SimpleNamespace as NS

    from compactor_vllm.core.model_runner import _check_shape_envelope

    cfg = NS(kvcache_page_size=128, leverage_sketch_size=48)
    _check_shape_envelope(NS(head_dim=128, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8), cfg)
    _check_shape_envelope(NS(head_dim=None, hidden_size=8192, num_attention_heads=64, num_key_value_heads=8), cfg)
    with pytest.raises(ValueError, match="head_dim 64"):
        _check_shape_envelope(NS(head_dim=64, hidden_size=2048, num_attention_heads=32, num_key_value_heads=8), cfg)
    with pytest.raises(ValueError, match="GQA group 16"):
        _check_shape_envelope(NS(head_dim=128, hidden_size=4096, num_attention_heads=32, num_key_value_heads=2), cfg)
    with pytest.raises(ValueError, match="page_size 64"):
        _check_shape_envelope(NS(head_dim=128, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8),
                              NS(kvcache_page_size=64, leverage_sketch_size=48))


def test_window_scorer_cuts_short_batches_into_one_wave():
    """CTAs of the SnapKV scorer that have keys, over calls of a few sequences: no second wave of CTAs for the sake of more
    splits, and no more splits than the workspace holds statistics of."""
    from compactor_vllm import _native as N

    for lens, heads in (([1220, 1987, 1640, 1076], 8), ([864, 1335, 1550, 1280, 1107, 1548], 8), ([8000] * 4, 8), ([500, 20000, 3000, 9000], 8),
                        ([2059, 1223, 2307], 8), ([8447, 6569, 3238, 9140, 3352], 4), ([40960], 8), ([1000], 8), ([300] * 9, 8)):
        for bound in (sum(lens), max(lens)):
            tiles = N.lib().cvllm_selftest_snap_split(len(lens), heads, sum(lens), bound)
            live = sum(-(-n // (128 * tiles)) for n in lens) * heads
            assert 0 < live <= 148, (lens, bound, tiles, live)
            splits = -(-bound // (128 * tiles))
            held = N.lib().cvllm_snapkv_scores_workspace_bytes(len(lens), bound, 4 * heads, heads, 32)
            assert len(lens) * heads * 2 * splits * 128 * 2 * 4 <= held
    assert N.lib().cvllm_selftest_snap_split(10, 8, 10000, 1000) == 8      # pairs enough: the fixed split
    assert N.lib().cvllm_selftest_snap_split(1, 8, 1000, 1000) == 1


def test_fields_of_a_parametrized_attention():
    """The attention's shortcut past Module.__getattr__ finds what the attribute finds, a parametrized weight too."""
    import torch
    from torch.nn.utils import parametrize

    from compactor_vllm.layers.attention import BiasedChunkAttention

    class Twice(torch.nn.Module):
        def forward(self, x):
            return 2 * x

    m = BiasedChunkAttention(4, 2, 64, 64, 0.125, qk_norm=True, sink=True, learned_sink=True, bucket_bias=(8, 64))
    names = ("inv_freq", "q_norm_weight", "k_norm_weight", "dist_bias", "rel", "slopes", "sink_logits")
    for name in names:
        assert m._field(name) is getattr(m, name), name
    for name in ("q_norm_weight", "sink_logits"):
        parametrize.register_parametrization(m, name, Twice())
        with torch.no_grad():
            m.parametrizations[name].original.fill_(3.0)
        assert torch.equal(m._field(name), getattr(m, name)) and (m._field(name) == 6.0).all(), name
    for name in names:
        assert (m._field(name) is None) == (getattr(m, name) is None), name


def test_remembered_sizes_are_per_device(monkeypatch):
    """A size that depends on the device's number of SMs is asked for once per device, on that device."""
    import contextlib

    from compactor_vllm import _native as N

    at, asked = [0], []

    class Library:
        def bytes(self, n):
            asked.append((at[0], n))
            return n * (100, 148)[at[0]]

    @contextlib.contextmanager
    def device(index):
        before, at[0] = at[0], index
        yield
        at[0] = before

    monkeypatch.setattr(N, "lib", Library)
    monkeypatch.setattr(N.torch.cuda, "device", device)
    N.sized.cache_clear()
    assert [N.sized(0, "bytes", 2), N.sized(1, "bytes", 2), N.sized(0, "bytes", 2), N.sized(1, "bytes", 3)] == [200, 296, 200, 444]
    assert asked == [(0, 2), (1, 2), (1, 3)]
    N.sized.cache_clear()


def test_heads_of_64_stream_from_where_it_pays():
    import torch

    from compactor_vllm.layers.attention import BiasedChunkAttention

    def choice(heads, kv, dim, keys, batch, **kw):
        m = BiasedChunkAttention(heads, kv, dim, dim, dim ** -0.5, **kw)
        m.k_cache, m.page_size = torch.empty(0, dim, dtype=torch.bfloat16), 128
        return m.streaming_decode_kernel(keys, batch)

    assert [choice(32, 8, 64, 256, b) for b in (1, 16, 24, 25, 32)] == [True, True, True, False, False]
    assert [choice(32, 8, 64, k, 32) for k in (319, 320)] == [False, True]
    assert [choice(32, 8, 64, k, 512) for k in (511, 512)] == [False, True]
    assert choice(32, 8, 128, 256, 512) and not choice(32, 8, 128, 255, 1)
    assert not choice(32, 8, 128, 4096, 513)          # more heads than its split covers
    assert choice(32, 8, 128, 4096, 1, window=128, keep_first=128) and not choice(32, 8, 128, 4096, 1, window=128)

"""Cases whose time is measured: the single steps of a served layer, each through the entry point that a program calls.

Kinds, and what each stands for in use:

  prefill    causal attention of new tokens over [paged, head-sparse prefix || new keys]: one long prompt, a ragged batch
             that continues from a compressed cache, a batch of short prompts
  decode     one query per sequence over the paged cache, ragged per (sequence, head)
  compactor  both scorers of COMPACTOR on a prompt or a packed batch of prompts (leverage of the keys before the rotation,
             attention mass inside chunks after it, blended), as the engine calls them: chunks of 512 and 128
  snapkv     the observation-window scorer of SnapKV
  evict      selection of the best (token, head) pairs per sequence and their compaction into the paged cache
  portion    a step of attention with biases, sinks, windows or rotation (`BiasedChunkAttention`) over portions of prompts
  step       the same attention, one token per sequence
  delta      the gated delta rule mixer over portions of prompts, or one token per sequence

Sizes are those of the repository's tests and benchmark (32 query and 8 key/value heads of 128 numbers, the shards of a
64-head model, pages of 128 tokens) and others of the same range.  A case is plain values; `lens` holds the new tokens of
every sequence.  Lengths that differ per (sequence, head) are a fixed function of the case, contents come from the seed.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "compactor-vllm_b200"))

from compactor_vllm.attention.sparse_decode_kernel import head_sparse_decode_attention  # noqa: E402
from compactor_vllm.attention.sparse_varlen_kernel import causal_sparse_varlen_with_cache  # noqa: E402
from compactor_vllm.compression.common import extract_and_store_top_kv  # noqa: E402
from compactor_vllm.compression.compactor import approximate_leverage_scores, non_causal_attn_scores  # noqa: E402
from compactor_vllm.compression.snapkv import query_aware_key_scores  # noqa: E402
from compactor_vllm.layers.attention import (BiasedChunkAttention, distance_buckets, linear_bias_slopes,  # noqa: E402
                                             pair_rotation_frequencies)
from compactor_vllm.layers.recurrent import DeltaRuleMixer  # noqa: E402
from compactor_vllm.utils import arguments  # noqa: E402
from compactor_vllm.utils.context import set_context  # noqa: E402

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
F64 = torch.float64
SKETCH, LEVERAGE_CHUNK, SCORE_CHUNK, WINDOW = 48, 512, 128, 32
PROTECTED_FIRST, PROTECTED_LAST = 16, 64
STYLES = ("slopes", "chunked", "window", "rotated")


def listed():
    return [
        # one long prompt: the largest piece of work of a served layer
        dict(name="prefill_32k", kind="prefill", lens="32768", prefix=0, hq=32, hkv=8, dtype="bf16"),
        # a ragged batch whose sequences continue from caches that were compressed unevenly per head
        dict(name="prefill_ragged", kind="prefill", lens="4000,2077,911,3301", prefix=2900, hq=32, hkv=8, dtype="bf16"),
        # short chat prompts on one shard of a 64-head model
        dict(name="prefill_short", kind="prefill", lens="17,64,129,33,200,90,31,256", prefix=0, hq=16, hkv=2, dtype="fp16"),
        # one user on a 16K context of which half is kept
        dict(name="decode_one", kind="decode", batch=1, rows=8192, hq=32, hkv=8, dtype="bf16"),
        # sixteen users on 40K contexts of which a quarter is kept
        dict(name="decode_batch", kind="decode", batch=16, rows=10240, hq=32, hkv=8, dtype="bf16"),
        # a few users at the beginning of their answers
        dict(name="decode_short", kind="decode", batch=8, rows=384, hq=32, hkv=8, dtype="fp16"),
        # COMPACTOR on a 16K prompt
        dict(name="compactor_16k", kind="compactor", lens="16384", hq=32, hkv=8, dtype="bf16"),
        # SnapKV on a 40K prompt
        dict(name="snapkv_40k", kind="snapkv", lens="40960", hq=32, hkv=8, dtype="bf16"),
        # half of a ragged batch's pairs stored
        dict(name="evict_ragged", kind="evict", lens="9000,3500,12000,511", ratio=0.5, hq=32, hkv=8, dtype="bf16"),
        # a prompt through windowed attention with a learned bias per distance and a sink per head
        dict(name="portion_window", kind="portion", lens="4096", start=0, style="window", hq=32, hkv=8, dim=128, page=128),
        # eight users decoding with linear distance biases and a sink
        dict(name="step_slopes", kind="step", batch=8, rows=4096, style="slopes", hq=32, hkv=8, dim=128, page=128),
        # a prompt through the gated delta rule
        dict(name="delta_4k", kind="delta", lens="4096", start=0, heads=32, kv_heads=16, dim=128, width=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, total, most):
    """`total` tokens over 1 .. most ragged sequences."""
    n = rng.randint(1, max(1, min(most, total)))
    w = [rng.uniform(0.2, 1.0) for _ in range(n)]
    lens = [max(1, int(total * x / sum(w))) for x in w]
    return ",".join(str(x) for x in lens)


def draw(rng):
    """Another case: a kind with the weight that it has among the listed ones, sizes over the range of use."""
    kind = rng.choice([c["kind"] for c in listed()])
    hq, hkv = rng.choice([(32, 8), (32, 8), (16, 2), (16, 4), (8, 1), (16, 8)])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "prefill":
        prefix = rng.choice([0, _log_int(rng, 50, 8000)])
        return dict(kind=kind, lens=_split(rng, _log_int(rng, 100, 24000), 16), prefix=prefix, hq=hq, hkv=hkv, dtype=dtype)
    if kind == "decode":
        batch = _log_int(rng, 1, 64)
        most = min(32768, 1200000 // (batch * hkv))
        return dict(kind=kind, batch=batch, rows=_log_int(rng, min(100, most), most), hq=hq, hkv=hkv, dtype=dtype)
    if kind in ("compactor", "snapkv"):
        lens = _split(rng, _log_int(rng, 600, 36000), 6)
        if kind == "compactor":
            # the Gram matrix of a tail shorter than the sketch is singular: its scores are rounding noise in any precision
            lens = ",".join(str(n + 96 if 0 < n % LEVERAGE_CHUNK < 96 else n) for n in map(int, lens.split(",")))
        return dict(kind=kind, lens=lens, hq=hq, hkv=hkv, dtype=dtype)
    if kind == "evict":
        return dict(kind=kind, lens=_split(rng, _log_int(rng, 600, 36000), 6), ratio=round(rng.uniform(0.1, 0.9), 2), hq=hq,
                    hkv=hkv, dtype=dtype)
    style, dim, page = rng.choice(STYLES), rng.choice([128, 128, 128, 64]), rng.choice([128, 128, 64])
    if kind == "portion":
        return dict(kind=kind, lens=_split(rng, _log_int(rng, 100, 8000), 6), start=rng.choice([0, _log_int(rng, 30, 4000)]),
                    style=style, hq=hq, hkv=hkv, dim=dim, page=page)
    if kind == "step":
        batch = _log_int(rng, 1, 32)
        most = min(16384, 800000 // (batch * hkv))
        return dict(kind=kind, batch=batch, rows=_log_int(rng, 60, most), style=style, hq=hq, hkv=hkv, dim=dim, page=page)
    heads, kv_heads = rng.choice([(32, 16), (16, 16), (16, 8), (32, 32)])
    dim = rng.choice([128, 128, 64])
    if rng.random() < 0.3:
        return dict(kind=kind, lens=",".join(["1"] * _log_int(rng, 1, 32)), start=rng.randint(5, 5000), heads=heads,
                    kv_heads=kv_heads, dim=dim, width=heads * dim)
    return dict(kind=kind, lens=_split(rng, _log_int(rng, 60, 6000), 6), start=0, heads=heads, kv_heads=kv_heads, dim=dim,
                width=heads * dim)


# ------------------------------------------------------------------ shapes

def _lens(case):
    return [int(x) for x in str(case["lens"]).split(",")]


def _spread(b, h):
    """A fixed number in [0, 1) per (sequence, head)."""
    return ((b * 7919 + h * 104729 + 37) * 2654435761 % 4294967296) / 4294967296.0


def _prefix_lens(case):
    return [[int(case["prefix"] * (0.3 + 0.9 * _spread(b, h))) for h in range(case["hkv"])] for b in range(len(_lens(case)))]


def _decode_lens(case):
    return [[max(1, int(case["rows"] * (0.5 + _spread(b, h)))) for h in range(case["hkv"])] for b in range(case["batch"])]


def _positions(case):
    """Position of the decoded token of every sequence."""
    return [max(0, int(case["rows"] * (0.6 + 0.8 * _spread(b, 0))) - 1) for b in range(case["batch"])]


def _cu(lens):
    out = [0]
    for n in lens:
        out.append(out[-1] + n)
    return out


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def _paged(g, pages_per_head, batch, hkv, dim, page, dtype, fill):
    """A paged cache as the engine's manager lays it out: one flat buffer each, physical pages in any order, slot 0
    reserved, the sequences in slots 1 .. batch.  `fill`: with normal numbers, else zeros."""
    n = (batch + 1) * hkv * pages_per_head
    table = torch.randperm(n, generator=g, device=DEV).to(torch.int32).view(batch + 1, hkv, pages_per_head).contiguous()
    shape = (n * page, dim)
    if not fill:
        return torch.zeros(shape, dtype=dtype, device=DEV), torch.zeros(shape, dtype=dtype, device=DEV), table
    return (torch.empty(shape, dtype=dtype, device=DEV).normal_(generator=g),
            torch.empty(shape, dtype=dtype, device=DEV).normal_(generator=g), table)


def _packed_qkv(g, n, hq, hkv, dim, dtype):
    """q, k, v as the model hands them over: views into one packed projection."""
    rows = _randn(g, n, (hq + 2 * hkv) * dim, dtype=dtype)
    return (rows[:, :hq * dim].view(n, hq, dim), rows[:, hq * dim:(hq + hkv) * dim].view(n, hkv, dim),
            rows[:, (hq + hkv) * dim:].view(n, hkv, dim))


def _rows_of(table, slot, h, n, page):
    pos = torch.arange(n, device=DEV)
    return table[slot, h, pos // page].long() * page + pos % page


# ------------------------------------------------------------------ prepare

def _prepare_prefill(case, g):
    lens, dt = _lens(case), DTYPES[case["dtype"]]
    hq, hkv, n = case["hq"], case["hkv"], sum(_lens(case))
    q, k, v = _packed_qkv(g, n, hq, hkv, 128, dt)
    s = dict(q=q, k=k, v=v, cu=_i32(_cu(lens)), max_q=max(lens), hkv=hkv, mapping=_i32(list(range(1, len(lens) + 1))))
    pl = _prefix_lens(case)
    most = max(max(r) for r in pl)
    s["kc"], s["vc"], s["table"] = _paged(g, most // 128 + 1, len(lens), hkv, 128, 128, dt, True)
    s["seq"], s["max_c"] = _i32(pl), most
    return s


def _prepare_decode(case, g):
    dt, dl = DTYPES[case["dtype"]], _decode_lens(case)
    most = max(max(r) for r in dl)
    s = dict(q=_randn(g, case["batch"], case["hq"], 128, dtype=dt), hkv=case["hkv"], seq=_i32(dl),
             mapping=_i32(list(range(1, case["batch"] + 1))))
    s["kc"], s["vc"], s["table"] = _paged(g, most // 128 + 1, case["batch"], case["hkv"], 128, 128, dt, True)
    return s


def _keys_like_a_models(g, n, hkv, dtype):
    """Keys before the rotation: a slow drift shared by the heads' numbers under noise."""
    pos = torch.linspace(0, 40.0, n, device=DEV)[:, None, None]
    low = 0.5 * torch.sin(pos + torch.arange(128, device=DEV) * 0.1) + _randn(g, 1, hkv, 128, scale=0.2)
    return (low + _randn(g, n, hkv, 128)).to(dtype)


def _prepare_scores(case, g):
    lens, dt = _lens(case), DTYPES[case["dtype"]]
    q, k, v = _packed_qkv(g, sum(lens), case["hq"], case["hkv"], 128, dt)
    s = dict(q=q, k=k, v=v, cu=_i32(_cu(lens)), max_q=max(lens), lens=lens)
    if case["kind"] == "compactor":
        q.mul_(128 ** -0.5)       # COMPACTOR takes the chunk's softmax unscaled: logits of a model's size
        s["k_pre"] = _keys_like_a_models(g, sum(lens), case["hkv"], dt)
        s["phi"] = arguments.make_phi(128, SKETCH, dt, DEV)
        s["first"], s["last"] = [PROTECTED_FIRST] * len(lens), [PROTECTED_LAST] * len(lens)
    return s


def _prepare_evict(case, g):
    lens, dt, hkv = _lens(case), DTYPES[case["dtype"]], case["hkv"]
    b = len(lens)
    _, k, v = _packed_qkv(g, sum(lens), case["hq"], hkv, 128, dt)
    scores = _randn(g, sum(lens), hkv)
    for i, n in zip(_cu(lens), lens):
        scores[i:min(i + PROTECTED_FIRST, i + n)] = math.inf
        scores[max(i, i + n - PROTECTED_LAST):i + n] = math.inf
    retain = arguments.tokens_to_retain(lens, [case["ratio"]] * b, [PROTECTED_FIRST] * b, [PROTECTED_LAST] * b, hkv)
    s = dict(k=k, v=v, scores=scores, cu=_i32(_cu(lens)), max_k=max(lens), hkv=hkv, retain=_i32(retain),
             top_k=arguments.max_tokens_to_retain(lens, hkv), mapping=_i32(list(range(1, b + 1))),
             empty=torch.zeros((b, hkv), dtype=torch.int32, device=DEV))
    s["kc"], s["vc"], s["table"] = _paged(g, max(lens) // 128 + 2, b, hkv, 128, 128, dt, False)
    return s


def _biased(case, g):
    """The attention of one layer, its cache behind it."""
    hq, hkv, dim, style = case["hq"], case["hkv"], case["dim"], case["style"]
    kw = dict(qk_norm=True, sink=True)
    if style == "slopes":
        kw.update(slopes=linear_bias_slopes(hq))
    elif style == "chunked":
        kw.update(slopes=linear_bias_slopes(hq), chunk=1024)
    elif style == "window":
        kw.update(window=1024, bucket_bias=(32, 1024), learned_sink=True)
    else:
        kw.update(rotation=pair_rotation_frequencies(64, 10000.0), learned_sink=True)
    a = BiasedChunkAttention(hq, hkv, dim, dim, dim ** -0.5, **kw).to(DEV)
    with torch.no_grad():
        for p in (a.q_norm_weight, a.k_norm_weight):
            p.copy_(1.0 + 0.1 * _randn(g, dim))
        if a.sink_logits is not None:
            a.sink_logits.copy_(_randn(g, hq))
        if a.rel is not None:
            a.refresh_distance_bias(_randn(g, 32, hq, scale=0.5))
    a.requires_grad_(False)
    return a


def _prepare_attention(case, g):
    hq, hkv, dim, page, dt = case["hq"], case["hkv"], case["dim"], case["page"], torch.bfloat16
    a = _biased(case, g)
    if case["kind"] == "portion":
        lens = _lens(case)
        starts = [int(case["start"] * (0.5 + _spread(b, 1))) for b in range(len(lens))]
    else:
        starts = _positions(case)
        lens = [1] * len(starts)
    ends = [x + n for x, n in zip(starts, lens)]
    b = len(lens)
    a.k_cache, a.v_cache, a.page_table = _paged(g, max(ends) // page + 1, b, hkv, dim, page, dt, True)
    a.bh_seq_lens = torch.zeros((b + 1, hkv), dtype=torch.int32, device=DEV)
    a.page_size = page
    positions = [p for x, n in zip(starts, lens) for p in range(x, x + n)]
    slots = [i + 1 for i, n in enumerate(lens) for _ in range(n)]
    ctx = dict(is_prefill=case["kind"] == "portion", cu_seqlens_q=_i32(_cu(lens)), cu_seqlens_k=_i32(_cu(lens)),
               max_seqlen_q=max(lens), max_seqlen_k=max(ends), batch_mapping=_i32(list(range(1, b + 1))),
               positions_i32=_i32(positions), token_slot=_i32(slots), seq_start=_i32(starts))
    return dict(attn=a, ctx=ctx, qkv=_randn(g, sum(lens), (hq + 2 * hkv) * dim, dtype=dt), starts=starts, lens=lens)


def _prepare_delta(case, g):
    lens, dt = _lens(case), torch.bfloat16
    heads, dim, width = case["heads"], case["dim"], case["width"]
    m = DeltaRuleMixer(width, heads, case["kv_heads"], dim, dim, 4, 1e-6).to(DEV)
    with torch.no_grad():
        m.conv_weight.copy_(_randn(g, *m.conv_weight.shape, scale=0.5))
        # step sizes from 1e-3 to 1e-1 and rates from 1 to 16, as such layers start
        dt0 = torch.exp(torch.rand(heads, generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))
        m.dt_bias.copy_(torch.log(torch.expm1(dt0)))
        m.A_log.copy_(torch.log(1.0 + 15.0 * torch.rand(heads, generator=g, device=DEV)))
        m.norm_weight.copy_(1.0 + 0.1 * _randn(g, dim))
    m.requires_grad_(False)
    m.o_proj = m.o_proj.to(dt)
    m.o_proj.weight.normal_(std=(heads * dim) ** -0.5, generator=g)
    state = m.make_state()
    b = len(lens)
    for name, (shape, kind) in state.state_specs(dt).items():
        setattr(state, name, _randn(g, b + 1, *shape, dtype=kind, scale=0.1 if name == "matrix_state" else 1.0))
    starts = [case["start"]] * b
    ctx = dict(is_prefill=max(lens) > 1, cu_seqlens_q=_i32(_cu(lens)), max_seqlen_q=max(lens),
               batch_mapping=_i32(list(range(1, b + 1))), seq_start=_i32(starts), positions_i32=_i32(starts) if max(lens) == 1 else
               _i32([p for x, n in zip(starts, lens) for p in range(x, x + n)]))
    cols = _randn(g, sum(lens), m.in_cols, dtype=dt)
    return dict(mixer=m, state=state, ctx=ctx, cols=cols, lens=lens)


PREPARE = {"prefill": _prepare_prefill, "decode": _prepare_decode, "compactor": _prepare_scores, "snapkv": _prepare_scores,
           "evict": _prepare_evict, "portion": _prepare_attention, "step": _prepare_attention, "delta": _prepare_delta}


def prepare(case, seed):
    with torch.no_grad():
        s = PREPARE[case["kind"]](case, _gen(seed))
    s["kind"] = case["kind"]
    return s


# ------------------------------------------------------------------ run

def _run_prefill(s):
    return causal_sparse_varlen_with_cache(
        s["q"], s["k"], s["v"], s["kc"], s["vc"], seq_lens_bh=s["seq"], global_page_table=s["table"],
        batch_mapping=s["mapping"], cu_seqlens_q=s["cu"], max_seqlen_q=s["max_q"], max_seqlen_k_cache=s["max_c"],
        HKV=s["hkv"], PAGE_SIZE=128, sm_scale=128 ** -0.5)


def _run_decode(s):
    return head_sparse_decode_attention(s["q"], s["kc"], s["vc"], s["seq"], s["table"], s["mapping"], s["hkv"], 128,
                                        128 ** -0.5)


def _run_compactor(s):
    pre = approximate_leverage_scores(s["k_pre"], s["lens"], s["phi"], normalize=True, chunk_size=LEVERAGE_CHUNK)
    return pre, non_causal_attn_scores(
        s["q"], s["k"], s["v"], s["cu"], s["max_q"], chunk_size=SCORE_CHUNK, sm_scale=1.0, normalize=True,
        accum_scores=pre, context_lens=s["lens"], protected_first_tokens=s["first"], protected_last_tokens=s["last"],
        accum_blending=0.5)


def _run_snapkv(s):
    return query_aware_key_scores(s["q"], s["k"], s["cu"], s["cu"], w=WINDOW)


def _run_evict(s):
    lens = s["empty"].clone()
    extract_and_store_top_kv(
        scores=s["scores"], cu_seqlens_k=s["cu"], max_k_len=s["max_k"], top_k=s["top_k"], H=s["hkv"], new_keys=s["k"],
        new_vals=s["v"], num_tokens_to_retain=s["retain"], page_table=s["table"], batch_mapping=s["mapping"], bh_lens=lens,
        k_cache=s["kc"], v_cache=s["vc"], PAGE_SIZE=128, PAD_TO_PAGE_SIZE=True)
    return lens, s["kc"], s["vc"]


def _run_attention(s):
    set_context(**s["ctx"])
    out = s["attn"](s["qkv"])
    return out, s["attn"].k_cache, s["attn"].v_cache, s["attn"].bh_seq_lens


def _run_delta(s):
    set_context(**s["ctx"])
    out = s["mixer"](None, s["cols"], s["state"])
    return out, s["state"].matrix_state, s["state"].conv_state


RUN = {"prefill": _run_prefill, "decode": _run_decode, "compactor": _run_compactor, "snapkv": _run_snapkv,
       "evict": _run_evict, "portion": _run_attention, "step": _run_attention, "delta": _run_delta}


def run(state):
    with torch.no_grad():
        return RUN[state["kind"]](state)


# ------------------------------------------------------------------ work

def _seen(case, i):
    """Keys that a query at position i sees."""
    if case["style"] == "chunked":
        return i % 1024 + 1
    return min(i + 1, 1024) if case["style"] == "window" else i + 1


def _seen_sum(case, start, n):
    if case["style"] in ("chunked", "window"):
        return sum(_seen(case, i) for i in range(start, start + n))
    return n * start + n * (n + 1) // 2


def work(case):
    kind, d = case["kind"], 128
    if kind == "prefill":
        lens, pl, hq, hkv = _lens(case), _prefix_lens(case), case["hq"], case["hkv"]
        pairs = sum(n * c + n * (n + 1) // 2 for n, row in zip(lens, pl) for c in row)
        rows = sum(sum(r) for r in pl)
        return {"bytes": 2 * d * (2 * sum(lens) * (hq + hkv) + 2 * rows), "flops": 4 * d * (hq // hkv) * pairs}
    if kind == "decode":
        rows = sum(sum(r) for r in _decode_lens(case))
        return {"bytes": 2 * d * (2 * rows + 2 * case["batch"] * case["hq"]), "flops": 4 * d * (case["hq"] // case["hkv"]) * rows}
    if kind in ("compactor", "snapkv", "evict"):
        lens, hq, hkv = _lens(case), case["hq"], case["hkv"]
        n, g = sum(lens), hq // hkv
        if kind == "compactor":
            pairs = sum((m // SCORE_CHUNK) * SCORE_CHUNK ** 2 + (m % SCORE_CHUNK) ** 2 for m in lens)
            return {"bytes": 2 * d * n * (hq + 2 * hkv) + 6 * n * hkv,
                    "flops": 2 * n * hkv * SKETCH * (d + 2 * SKETCH) + 2 * d * hq * pairs}
        if kind == "snapkv":
            far = sum(max(m - WINDOW, 0) for m in lens)
            return {"bytes": 2 * d * (far * hkv + len(lens) * WINDOW * hq) + 4 * n * hkv,
                    "flops": 2 * d * WINDOW * g * hkv * far}
        b = len(lens)
        kept = sum(arguments.tokens_to_retain(lens, [case["ratio"]] * b, [PROTECTED_FIRST] * b, [PROTECTED_LAST] * b, hkv))
        return {"bytes": 4 * n * hkv + 2 * 2 * 2 * d * kept, "flops": 0}
    if kind in ("portion", "step"):
        hq, hkv, d = case["hq"], case["hkv"], case["dim"]
        if kind == "portion":
            lens = _lens(case)
            spans = [(int(case["start"] * (0.5 + _spread(b, 1))), n) for b, n in enumerate(lens)]
        else:
            spans = [(p, 1) for p in _positions(case)]
        new = sum(n for _, n in spans)
        # cached rows in front of a portion that its first query still sees
        old = sum(min(_seen(case, x) - 1, x) for x, n in spans)
        return {"bytes": 2 * d * (new * (hq + 2 * hkv) + new * 2 * hkv + new * hq + 2 * old * hkv),
                "flops": 4 * d * hq * sum(_seen_sum(case, x, n) for x, n in spans)}
    lens, heads, dim, width = _lens(case), case["heads"], case["dim"], case["width"]
    n, b = sum(lens), len(lens)
    cols = 2 * case["kv_heads"] * dim + 2 * heads * dim + 2 * heads
    state = 4 * b * heads * dim * dim * (2 if case["start"] else 1)
    return {"bytes": 2 * n * (cols + width) + 2 * heads * dim * width + state,
            "flops": 6 * n * heads * dim * dim + 2 * n * heads * dim * width}


# ------------------------------------------------------------------ tolerance

def tolerance(case):
    """About four times the distance from 64 bits (attention: that of a result rounded once to its type)."""
    kind = case["kind"]
    if kind == "evict":
        return "exact"            # rows are moved, not computed
    if kind == "compactor":
        return {"rel": 0.02, "max": 0.3}      # the sketch, its Gram matrix and its factors are rounded to 16 bits on the way
    if kind == "snapkv":
        return {"rel": 1e-5, "max": 1e-3}     # 32-bit sums
    return {"rel": 0.001 if case.get("dtype") == "fp16" else 0.008, "max": 0.2}


# ------------------------------------------------------------------ exact

def _attend64(q, k, v, scale, start, bias=None, seen=None, sink=None):
    """q [n, D] at positions start .. start + n - 1 of one head against k, v [m, D] at positions 0 .. m - 1, in 64 bits.
    bias(dist) and seen(i, j) take matrices of distances and positions; sink: an extra score without a value."""
    out = torch.empty(q.shape[0], v.shape[1], dtype=F64, device=DEV)
    step = max(64, (1 << 27) // max(1, k.shape[0]))
    j = torch.arange(k.shape[0], device=DEV)[None]
    for a in range(0, q.shape[0], step):
        i = torch.arange(start + a, start + min(a + step, q.shape[0]), device=DEV)[:, None]
        last = int(i[-1]) + 1
        s = (q[a:a + step] @ k[:last].T).mul_(scale)
        jj = j[:, :last]
        if bias is not None:
            s += bias((i - jj).clamp_(min=0))
        s.masked_fill_((jj > i) if seen is None else ((jj > i) | ~seen(i, jj)), -math.inf)
        top = s.amax(dim=-1, keepdim=True)
        if sink is not None:
            top = top.clamp(min=float(sink))
        s.sub_(top).exp_()
        den = s.sum(dim=-1, keepdim=True)
        if sink is not None:
            den += torch.exp(float(sink) - top)
        out[a:a + step] = (s @ v[:last]) / den
    return out


def _exact_prefill(case, s):
    lens, pl = _lens(case), _prefix_lens(case)
    hq, hkv = case["hq"], case["hkv"]
    cu, per = _cu(lens), case["hq"] // case["hkv"]
    out = torch.empty(sum(lens), hq, 128, dtype=F64, device=DEV)
    for b, n in enumerate(lens):
        at = slice(cu[b], cu[b] + n)
        for h in range(hkv):
            c = pl[b][h]
            rows = _rows_of(s["table"], b + 1, h, c, 128)
            k = torch.cat([s["kc"][rows], s["k"][at, h]]).to(F64)
            v = torch.cat([s["vc"][rows], s["v"][at, h]]).to(F64)
            for x in range(h * per, (h + 1) * per):
                out[at, x] = _attend64(s["q"][at, x].to(F64), k, v, 128 ** -0.5, c)
    return out


def _exact_decode(case, s):
    per = case["hq"] // case["hkv"]
    out = torch.empty(case["batch"], case["hq"], 128, dtype=F64, device=DEV)
    for b, row in enumerate(_decode_lens(case)):
        for h, n in enumerate(row):
            rows = _rows_of(s["table"], b + 1, h, n, 128)
            x = slice(h * per, (h + 1) * per)
            p = torch.softmax(s["q"][b, x].to(F64) @ s["kc"][rows].to(F64).T * 128 ** -0.5, dim=-1)
            out[b, x] = p @ s["vc"][rows].to(F64)
    return out


def _zscore64(x):
    return (x - x.mean()) / x.var(unbiased=False).sqrt()


def _exact_compactor(case, s):
    lens, hq, hkv = _lens(case), case["hq"], case["hkv"]
    pre = torch.empty(sum(lens), hkv, dtype=F64, device=DEV)
    post = torch.empty_like(pre)
    x = s["k_pre"].to(F64) @ s["phi"].to(F64)
    for b, (at, n) in enumerate(zip(_cu(lens), lens)):
        for c in range(at, at + n, LEVERAGE_CHUNK):
            e = min(c + LEVERAGE_CHUNK, at + n)
            y = x[c:e].transpose(0, 1)
            y = y - y.mean(dim=1, keepdim=True)
            gram = y.transpose(1, 2) @ y + 5e-3 * torch.eye(SKETCH, dtype=F64, device=DEV)
            lev = (torch.linalg.solve(gram, y.transpose(1, 2)) * y.transpose(1, 2)).sum(dim=1)
            pre[c:e] = _zscore64(lev.T)
        for c in range(at, at + n, SCORE_CHUNK):
            e = min(c + SCORE_CHUNK, at + n)
            q = s["q"][c:e].to(F64).view(e - c, hkv, hq // hkv, 128).permute(1, 0, 2, 3).reshape(hkv, -1, 128)
            p = torch.softmax(q @ s["k"][c:e].to(F64).permute(1, 2, 0), dim=-1)
            # rows that fill up the last 64-row tile of a short chunk count 1 / chunk each
            post[c:e] = p.sum(dim=1).T + (-(e - c) % 64) * (hq // hkv) / SCORE_CHUNK
        sc = post[at:at + n]
        sc.copy_(_zscore64(sc) + 0.5 * pre[at:at + n])
        sc[:min(PROTECTED_FIRST, n)] = math.inf
        sc[max(0, n - PROTECTED_LAST):] = math.inf
    return pre, post


def _exact_snapkv(case, s):
    lens, hq, hkv = _lens(case), case["hq"], case["hkv"]
    out = torch.zeros(sum(lens), hkv, dtype=F64, device=DEV)
    for at, n in zip(_cu(lens), lens):
        far = n - WINDOW
        if far <= 0:
            continue
        q = s["q"][at + far:at + n].to(F64).view(WINDOW, hkv, hq // hkv, 128).permute(1, 0, 2, 3).reshape(hkv, -1, 128)
        p = torch.softmax(q @ s["k"][at:at + far].to(F64).permute(1, 2, 0) * 128 ** -0.5, dim=-1).sum(dim=1)   # [hkv, far]
        full = torch.nn.functional.pad(p, (0, -far % 64)).view(hkv, -1, 64)
        total = sum(torch.nn.functional.pad(full, (t, 0))[..., :64] for t in range(5))
        count = torch.arange(1, 65, device=DEV, dtype=F64).clamp(max=5)
        out[at:at + far] = (total / count).view(hkv, -1)[:, :far].T
        out[at + far:at + n] = math.inf
    return out


def _exact_attention(case, s):
    hq, hkv, dim, page, a = case["hq"], case["hkv"], case["dim"], case["page"], s["attn"]
    rows = s["qkv"].to(F64)
    n = rows.shape[0]

    def normed(x, w, pos):
        if case["style"] == "rotated":
            turn = pos.to(F64)[:, None] * a.inv_freq[None]
            c, z = torch.cos(turn)[:, None], torch.sin(turn)[:, None]
            m = 2 * a.inv_freq.numel()
            e, o = x[..., 0:m:2].clone(), x[..., 1:m:2].clone()
            x[..., 0:m:2], x[..., 1:m:2] = e * c - o * z, o * c + e * z
        return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + 1e-6) * w.to(F64)

    pos = s["ctx"]["positions_i32"]
    q = normed(rows[:, :hq * dim].reshape(n, hq, dim).clone(), a.q_norm_weight, pos)
    k = normed(rows[:, hq * dim:(hq + hkv) * dim].reshape(n, hkv, dim).clone(), a.k_norm_weight, pos)
    v = rows[:, (hq + hkv) * dim:].reshape(n, hkv, dim)
    out = torch.empty(n, hq, dim, dtype=F64, device=DEV)
    style, per = case["style"], hq // hkv
    slopes = linear_bias_slopes(hq)
    bucket = torch.tensor(distance_buckets(32, 1024, 1025), device=DEV)
    seen = None
    if style == "chunked":
        seen = lambda i, j: i // 1024 == j // 1024  # noqa: E731
    elif style == "window":
        seen = lambda i, j: i - j < 1024  # noqa: E731
    at = 0
    for b, (x, m) in enumerate(zip(s["starts"], s["lens"])):
        now = slice(at, at + m)
        for h in range(hkv):
            old = _rows_of(a.page_table, b + 1, h, x, page)
            kk = torch.cat([a.k_cache[old].to(F64), k[now, h]])
            vv = torch.cat([a.v_cache[old].to(F64), v[now, h]])
            for i in range(h * per, (h + 1) * per):
                bias = None
                if style in ("slopes", "chunked"):
                    bias = lambda d, i=i: d.to(F64) * -float(slopes[i])  # noqa: E731
                elif style == "window":
                    table = a.rel[:, i].to(F64)[bucket]
                    bias = lambda d, table=table: table[d.clamp(max=1024)]  # noqa: E731
                sink = 0.0 if a.sink_logits is None else float(a.sink_logits[i])
                out[now, i] = _attend64(q[now, i], kk, vv, dim ** -0.5, x, bias, seen, sink)
        at += m
    return out.view(n, hq * dim), None, None, None


def _exact_delta(case, s):
    m, st, lens = s["mixer"], s["state"], s["lens"]
    heads, kv, dim = case["heads"], case["kv_heads"], case["dim"]
    cols, taps = s["cols"].to(F64), m.taps
    c = m.conv_channels
    state = st.matrix_state.to(F64).clone()                       # [slots, heads, value, key]
    out = torch.empty(cols.shape[0], heads * dim, dtype=F64, device=DEV)
    at = 0
    for b, n in enumerate(lens):
        x = cols[at:at + n]
        before = st.conv_state[b + 1].to(F64) if case["start"] else torch.zeros(taps - 1, c, dtype=F64, device=DEV)
        raw = torch.cat([before, x[:, :c]])
        y = sum(raw[t:t + n] * m.conv_weight[:, t].to(F64) for t in range(taps))
        y = y * torch.sigmoid(y)
        q, k = (y[:, i * kv * dim:(i + 1) * kv * dim].view(n, kv, dim) for i in (0, 1))
        q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q, k = ((z * f).repeat_interleave(heads // kv, dim=1) for z, f in ((q, dim ** -0.5), (k, 1.0)))
        v = y[:, 2 * kv * dim:].view(n, heads, dim)
        g_off = c
        gate = x[:, g_off:g_off + heads * dim]
        beta = torch.sigmoid(x[:, g_off + heads * dim:g_off + heads * dim + heads])
        decay = torch.exp(-torch.exp(m.A_log.to(F64)) * torch.nn.functional.softplus(
            x[:, g_off + heads * dim + heads:] + m.dt_bias.to(F64), threshold=100.0))
        a = state[b + 1] if case["start"] else torch.zeros_like(state[b + 1])
        o = torch.empty(n, heads, dim, dtype=F64, device=DEV)
        for t in range(n):
            a = a * decay[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(a, k[t][:, :, None])[:, :, 0])
            a = torch.baddbmm(a, u[:, :, None], k[t][:, None])
            o[t] = torch.bmm(a, q[t][:, :, None])[:, :, 0]
        state[b + 1] = a
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * m.norm_weight.to(F64)
        out[at:at + n] = o.reshape(n, heads * dim) * gate * torch.sigmoid(gate)
        at += n
    return out @ m.o_proj.weight.to(F64).T, state, None


EXACT = {"prefill": _exact_prefill, "decode": _exact_decode, "compactor": _exact_compactor, "snapkv": _exact_snapkv,
         "portion": _exact_attention, "step": _exact_attention, "delta": _exact_delta}


def exact(case, seed):
    """The outputs in 64 bits from the same inputs, without this repository's kernels."""
    if case["kind"] not in EXACT:
        return None
    with torch.no_grad():
        return EXACT[case["kind"]](case, prepare(case, seed))

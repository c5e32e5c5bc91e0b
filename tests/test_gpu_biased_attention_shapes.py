"""Portions of the biased attention over the head sizes, page sizes and bias tables that its tensor-core kernel serves (and
their neighbours that it leaves to the others), against the formula in 64 bits.

Tolerance: scores are sums of exact 16-bit products in 32 bits, P and the result are rounded to bfloat16 once each (2^-9
relative, so 2^-9 / sqrt(3) root mean square each): 2.8e-3 relative in the 2-norm is the most that both leave; 6e-3 is
twice that."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def make(H, G, D, page, spans, seed, **kw):
    """A module with its cache: rows up to every sequence's last position written, all others NaN."""
    from compactor_vllm.layers.attention import BiasedChunkAttention

    g = torch.Generator().manual_seed(seed)
    with torch.device(DEV):
        m = BiasedChunkAttention(H, G, D, D, D ** -0.5, **kw).to(DEV)
    ends = [s + n for s, n in spans]
    B, P = len(spans), max(-(-e // page) for e in ends)
    rows = (B + 1) * G * P * page
    m.page_table = torch.randperm((B + 1) * G * P, generator=g).to(torch.int32).view(B + 1, G, P).to(DEV)
    m.k_cache = torch.full((rows, D), float("nan"), dtype=torch.bfloat16, device=DEV)
    m.v_cache = m.k_cache.clone()
    m.page_size = page
    keys = []
    for b, e in enumerate(ends):
        k, v = (torch.randn(e, G, D, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
        p = torch.arange(e, device=DEV)
        for h in range(G):
            at = m.page_table[b + 1, h].long()[p // page] * page + p % page
            m.k_cache[at], m.v_cache[at] = k[:, h], v[:, h]
        keys.append((k.double(), v.double()))
    q = torch.randn(sum(n for _, n in spans), H, D, generator=g).to(torch.bfloat16).to(DEV)
    return m, q, keys


def context(spans, decode):
    from compactor_vllm.utils.context import set_context

    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for _, n in spans:
        cu.append(cu[-1] + n)
    set_context(is_prefill=not decode, cu_seqlens_q=i32(cu), max_seqlen_q=max(n for _, n in spans),
                max_seqlen_k=max(s + n for s, n in spans), batch_mapping=i32(range(1, len(spans) + 1)),
                positions_i32=i32([p for s, n in spans for p in range(s, s + n)]), seq_start=i32([s for s, _ in spans]))


def formula(m, q, keys, spans):
    H, G, D = m.num_heads, m.num_kv_heads, m.head_dim
    out, at = [], 0
    for (k, v), (start, n) in zip(keys, spans):
        i = torch.arange(start, start + n, device=DEV)[:, None]
        j = torch.arange(k.shape[0], device=DEV)[None]
        ok = torch.ones_like(i - j, dtype=torch.bool)
        if m.chunk:
            ok &= i // m.chunk == j // m.chunk
        if m.window:
            ok &= i - j < m.window
        ok = (ok | (j < m.keep_first)) & (j <= i)
        kk, vv = (x.repeat_interleave(H // G, dim=1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[at:at + n].double(), kk) * m.scale
        dist = (i - j).clamp(min=0)
        if m.slopes is not None:
            s -= m.slopes.double()[:, None, None] * dist
        if m.dist_bias is not None:
            s += m.dist_bias.double()[dist.clamp(max=m.dist_bias.shape[0] - 1)].permute(2, 0, 1)
        s = s.masked_fill(~ok, -math.inf)
        sink = torch.full((H, n, 1), 0.0 if m.sink else -math.inf, dtype=torch.float64, device=DEV)
        if m.sink_logits is not None:
            sink += m.sink_logits.double()[:, None, None]
        p = torch.softmax(torch.cat([s, sink], dim=-1), dim=-1)[..., :-1]
        out.append(torch.einsum("hqk,khd->qhd", p, vv).reshape(n, H * D))
        at += n
    return torch.cat(out)


def options(seed, H, rows, slopes, sink, window, keep, chunk):
    from compactor_vllm.layers.attention import linear_bias_slopes

    kw = dict(window=window, keep_first=keep, chunk=chunk, sink=sink != "none", learned_sink=sink == "learned")
    if slopes:
        kw["slopes"] = linear_bias_slopes(H)
    return kw


def dress(m, rows, seed):
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        if m.sink_logits is not None:
            m.sink_logits.copy_(torch.randn(m.num_heads, generator=g))
    if rows:
        m.dist_bias = torch.randn(rows, m.num_heads, generator=g).to(DEV)
        m.rel = torch.nn.Parameter(m.dist_bias)


# portions that begin and end on and off the 128-row tiles and the pages, one of a single token
SPANS = [(0, 300), (255, 130), (640, 1), (511, 129), (129, 127)]

# H, G, D, page, table rows, slopes, sink, window, kept tokens, chunk
CASES = [
    (4, 2, 128, 128, 0, True, "zero", 0, 0, 0),
    (4, 2, 128, 128, 1, False, "learned", 0, 0, 0),
    (4, 2, 128, 128, 200, True, "none", 0, 0, 0),
    (4, 2, 128, 64, 130, False, "learned", 257, 0, 0),
    (2, 1, 128, 32, 700, True, "zero", 128, 5, 0),
    (2, 1, 128, 16, 0, True, "none", 0, 130, 200),
    (8, 1, 128, 256, 3584, False, "zero", 0, 0, 0),
    (2, 1, 128, 128, 3585, False, "zero", 0, 0, 0),      # a table past what lies in shared memory
    (4, 2, 64, 128, 0, False, "learned", 0, 0, 0),
    (4, 2, 64, 64, 90, True, "none", 0, 0, 0),
    (8, 2, 64, 32, 300, False, "zero", 100, 140, 0),
    (4, 2, 64, 16, 0, True, "zero", 0, 0, 300),
    (3, 1, 64, 64, 40, True, "zero", 0, 0, 0),           # an odd group
    (4, 2, 128, 48, 40, True, "zero", 0, 0, 0),          # pages that do not divide a tile
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_portions(case):
    from compactor_vllm.utils.context import reset_context

    H, G, D, page, rows, slopes, sink, window, keep, chunk = case
    m, q, keys = make(H, G, D, page, SPANS, 11, **options(1, H, rows, slopes, sink, window, keep, chunk))
    dress(m, rows, 2)
    context(SPANS, False)
    try:
        got = m.attend(q).double()
    finally:
        reset_context()
    want = formula(m, q, keys, SPANS)
    assert torch.isfinite(got).all()
    assert ((got - want).norm() / want.norm()).item() < 6e-3


@pytest.mark.parametrize("case", [c for c in CASES if c[4] <= 3584 and c[0] // c[1] % 2 == 0 and c[3] != 48],
                         ids=lambda c: "-".join(map(str, c)))
def test_portions_lose_no_precision(case):
    """The tensor-core kernel's distance from the formula beside the mma.sync kernel's, which served these shapes before it:
    both round P (the row's largest weight is 1 there, which rounding keeps) and the result to bfloat16.  The two errors are
    sums of the same kind over some 10^5 outputs, which agree within 0.5 % of each other by chance; an exponential good to
    1e-4 or a reference below the row's maximum costs 1 to 3 %.  Heads of 128 in whole pages without a table have always
    had both, and are left out."""
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context

    H, G, D, page, rows, slopes, sink, window, keep, chunk = case
    if D == 128 and not rows and page % 128 == 0:
        pytest.skip("always on the tensor-core kernel")
    spans = [(0, 700), (255, 330), (640, 400)]
    m, q, keys = make(H, G, D, page, spans, 17, **options(1, H, rows, slopes, sink, window, keep, chunk))
    dress(m, rows, 4)
    want = formula(m, q, keys, spans)
    errs = []
    for option in (0, 2):
        context(spans, False)
        N.set_test_option("bias_attn_fma", option)
        try:
            got = m.attend(q).double()
        finally:
            N.set_test_option("bias_attn_fma", 0)
            reset_context()
        errs.append(((got - want).norm() / want.norm()).item())
    print(case, errs)
    assert errs[0] <= 1.005 * errs[1], errs


# decoding: positions at and around unit, window and chunk borders, one at position 0, one on the reserved slot
DECODE = [(p, 1) for p in (0, 1, 127, 128, 255, 299, 300, 511, 640, 1100)]


def decode(m, q, option=0, spans=DECODE):
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import get_context, reset_context

    context(spans, True)
    get_context().batch_mapping[4] = 0       # a padding row
    N.set_test_option("bias_attn_fma", option)
    try:
        return m.attend(q).double()
    finally:
        N.set_test_option("bias_attn_fma", 0)
        reset_context()


@pytest.mark.parametrize("case", [c for c in CASES if c[1] * 8 >= c[0]] + [(16, 2, 128, 128, 50, True, "learned", 0, 0, 0),
                                                                           (5, 1, 64, 64, 0, True, "zero", 200, 3, 0)],
                         ids=lambda c: "-".join(map(str, c)))
def test_decoding(case):
    """The streaming kernel keeps P in 32 bits (as two 16-bit parts), so only the result's rounding is left: 2^-9 / sqrt(3)
    = 1.2e-3; 2.5e-3 is twice that.  It is no further from the formula than the FMA kernel, whose P is one 32-bit number."""
    H, G, D, page, rows, slopes, sink, window, keep, chunk = case
    m, q, keys = make(H, G, D, page, DECODE, 12, **options(1, H, rows, slopes, sink, window, keep, chunk))
    dress(m, rows, 3)
    want = formula(m, q, keys, DECODE)
    want[4] = 0
    err = lambda x: ((x - want).norm() / want.norm()).item()
    got, fma = decode(m, q), decode(m, q, 1)
    assert torch.isfinite(got).all() and (got[4] == 0).all()
    assert err(got) < 2.5e-3 and err(got) < 1.05 * err(fma) + 1e-6


def test_decoding_far_sinks_and_scores():
    """Sinks far above and far below every key, scores large enough that only the running maximum keeps them finite."""
    m, q, keys = make(4, 2, 128, 128, DECODE, 13, sink=True, learned_sink=True)
    q = (q * 8).contiguous()
    with torch.no_grad():
        m.sink_logits.copy_(torch.tensor([500.0, -500.0, 60.0, 0.0]))
    want = formula(m, q, keys, DECODE)
    want[4] = 0
    got = decode(m, q)
    assert torch.isfinite(got).all()
    assert ((got - want).norm() / want.norm()).item() < 2.5e-3


# whole units lie between the kept tokens and the window or the chunk of the last ones
KEPT = [(p, 1) for p in (0, 255, 256, 383, 511, 640, 767, 1100, 1535, 1900)]


@pytest.mark.parametrize("window,keep,chunk", [(256, 5, 0), (300, 130, 0), (256, 400, 0), (0, 140, 256), (700, 3, 512), (257, 1, 0)])
@pytest.mark.parametrize("D,page", [(128, 128), (128, 64), (64, 128), (64, 16)])
def test_decoding_with_kept_tokens(D, page, window, keep, chunk):
    """Kept first tokens on the streaming kernel: fewer than a unit, several units, up to and into the window's first."""
    m, q, keys = make(8, 2, D, page, KEPT, 14, **options(1, 8, 60, True, "zero", window, keep, chunk))
    dress(m, 60, 5)
    assert m.streaming_decode_kernel(1901)
    want = formula(m, q, keys, KEPT)
    want[4] = 0
    err = lambda x: ((x - want).norm() / want.norm()).item()
    got = decode(m, q, spans=KEPT)
    assert torch.isfinite(got).all() and (got[4] == 0).all()
    assert err(got) < 2.5e-3 and err(got) < 1.05 * err(decode(m, q, 1, KEPT)) + 1e-6


@pytest.mark.parametrize("H,G,D", [(8, 1, 128), (16, 2, 64)])
@pytest.mark.parametrize("units", [9, 40, 68, 69, 70, 142, 143, 144, 160])
def test_decoding_cut_heads(H, G, D, units):
    """A long sequence beside three short ones, (units + 5) G units in all: fewer than CTAs (148), as many, more."""
    spans = [(0, 1), (128 * units - 1, 1), (127, 1), (300, 1), (700, 1)]
    m, q, keys = make(H, G, D, 128, spans, units, **options(1, H, 0, True, "zero", 0, 0, 0))
    want = formula(m, q, keys, spans)
    want[4] = 0
    got = decode(m, q, spans=spans)
    assert torch.isfinite(got).all() and (got[4] == 0).all()
    assert ((got - want).norm(dim=1) <= 2.5e-3 * want.norm(dim=1)).all()


def test_decode_kernel_does_not_depend_on_earlier_steps():
    """What a step runs on follows from the step: a step on three key splits gives the same bits before and after a step that
    left a large workspace behind, and those are not the streaming kernel's."""
    m, q, keys = make(8, 2, 128, 128, DECODE, 15, sink=True)
    streamed = decode(m, q)
    m.streaming_decode_kernel, m.decode_splits = lambda *_: False, lambda *_: 3
    before = decode(m, q)
    assert not torch.equal(before, streamed)
    long, q_long, _ = make(8, 2, 128, 128, [(300, 1)] * 150, 16, sink=True)
    context([(300, 1)] * 150, True)
    long.attend(q_long)
    assert torch.equal(decode(m, q), before)


def test_kept_tokens_count_for_the_choice_of_the_decode_kernel():
    m, q, keys = make(4, 2, 128, 128, [(40, 1)], 18, window=128, keep_first=512)
    assert m.streaming_decode_kernel(4096) and m.streaming_decode_kernel(256) and not m.streaming_decode_kernel(255)


@pytest.mark.parametrize("what", ["out", "query", "width"])
def test_decoding_into_rows_that_the_streaming_kernel_refuses(what):
    """Outputs off the 4-byte grid, at odd row strides, or queries off the 16-byte grid take the key splits, as many as
    the step's keys ask for."""
    from compactor_vllm.utils.context import reset_context

    m, q, keys = make(8, 2, 64, 64, DECODE, 19, sink=True)
    T, width = q.shape[0], 8 * 64
    if what == "query":
        flat = torch.zeros(q.numel() + 1, dtype=q.dtype, device=DEV)
        flat[1:] = q.flatten()
        q = flat[1:].view_as(q)
    rows = width + (1 if what == "width" else 2)
    out = torch.zeros(T * rows + 1, dtype=q.dtype, device=DEV)[1 if what == "out" else 0:][:T * rows].view(T, rows)[:, :width]
    want = formula(m, q, keys, DECODE)
    context(DECODE, True)
    asked = []
    splits = m.decode_splits
    m.decode_splits = lambda *a: asked.append(splits(*a)) or asked[-1]
    try:
        got = m.attend(q, out=out if what != "query" else None).double()
    finally:
        reset_context()
    assert asked and asked[0] > 1
    assert ((got - want).norm() / want.norm()).item() < 2.5e-3


@pytest.mark.parametrize("D,page,rows", [(128, 64, 0), (128, 128, 40), (64, 128, 0), (64, 16, 40)])
@pytest.mark.parametrize("window,keep,chunk", [(300, 0, 0), (300, 5, 0), (0, 130, 256)])
def test_values_that_no_row_sees(D, page, rows, window, keep, chunk):
    """Values outside every query's window or chunk that share a tile with seen ones may be infinite or NaN."""
    from compactor_vllm.utils.context import reset_context

    start, n = 1100, 50
    m, q, keys = make(4, 2, D, page, [(start, n)], 21, **options(1, 4, rows, False, "zero", window, keep, chunk))
    dress(m, rows, 6)
    (k, v), p = keys[0], torch.arange(start + n, device=DEV)
    seen = p >= (start - window + 1 if window else start // chunk * chunk)
    hidden = p[~seen & (p >= keep)]
    for h in range(2):
        at = m.page_table[1, h].long()[hidden // page] * page + hidden % page
        m.v_cache[at] = torch.tensor([math.inf, math.nan, -math.inf], device=DEV).to(torch.bfloat16)[hidden % 3][:, None]
    want = formula(m, q, keys, [(start, n)])
    context([(start, n)], False)
    try:
        got = m.attend(q).double()
    finally:
        reset_context()
    assert torch.isfinite(got).all()
    assert ((got - want).norm() / want.norm()).item() < 6e-3
    last = [(start + n - 1, 1)]
    got, want = decode_one(m, q[-1:].contiguous(), last), formula(m, q[-1:].contiguous(), keys, last)
    assert ((got - want).norm() / want.norm()).item() < 2.5e-3


def decode_one(m, q, spans):
    from compactor_vllm.utils.context import reset_context

    context(spans, True)
    try:
        return m.attend(q).double()
    finally:
        reset_context()


@pytest.mark.parametrize("D,page", [(128, 64), (64, 128)])
def test_scores_far_below(D, page):
    """Scores of -10^32 are scores: they weigh nothing beside others and the same among themselves."""
    from compactor_vllm.utils.context import reset_context

    spans = [(0, 200), (300, 90)]
    m, q, keys = make(4, 2, D, page, spans, 22)
    m.dist_bias = torch.zeros(150, 4, device=DEV)
    m.dist_bias[:140] = -1e32
    m.rel = torch.nn.Parameter(m.dist_bias)
    context(spans, False)
    try:
        got = m.attend(q).double()
    finally:
        reset_context()
    want = formula(m, q, keys, spans)
    assert torch.isfinite(got).all()
    assert ((got - want).norm() / want.norm()).item() < 6e-3
    m.dist_bias[140:] = -1e32
    at = [(389, 1)]
    m2, q2, keys2 = make(4, 2, D, page, at, 23)
    m2.dist_bias, m2.rel = m.dist_bias, m.rel
    got, want = decode_one(m2, q2, at), formula(m2, q2, keys2, at)
    assert m2.streaming_decode_kernel(390)
    assert ((got - want).norm() / want.norm()).item() < 2.5e-3


@pytest.mark.parametrize("H,spans,latent", [(8, [(0, 2368)], True), (8, [(0, 2369)], False), (32, [(100, 300), (0, 200)], True),
                                            (32, [(0, 700)], False), (2, [(0, 90)], True)])
def test_rows_of_64_that_are_their_own_values(H, spans, latent):
    """One wave of packed query rows stays on the kernel for latent rows (option 3 asks for it everywhere), more do not."""
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context

    m, q, keys = make(H, 1, 64, 64, spans, 24, values_in_keys=True, sink=True)
    keys = [(k, k) for k, _ in keys]
    out = []
    for option in (0, 3):
        context(spans, False)
        N.set_test_option("bias_attn_fma", option)
        try:
            out.append(m.attend(q))
        finally:
            N.set_test_option("bias_attn_fma", 0)
            reset_context()
    assert torch.equal(*out) == latent
    want = formula(m, q, keys, spans)
    for got in out:
        assert ((got.double() - want).norm() / want.norm()).item() < 6e-3

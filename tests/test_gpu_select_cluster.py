"""Selection and compaction: the one-launch selection (a cluster per sequence) against the chain of launches, exactly, over
head counts, ragged batches, score strides, ties, infinities and NaN, and the sizes where clusters grow."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
D, PS = 64, 128


def scores_of(kind, n, H, g):
    s = torch.randn(n, H, generator=g)
    if kind == "ties":                       # a handful of values: nearly every threshold is a tie
        s = torch.randint(0, 5, (n, H), generator=g).float()
    elif kind == "equal":
        s.zero_()
    elif kind == "special":
        r = torch.rand(n, H, generator=g)
        s[r < 0.05] = float("inf")
        s[(r >= 0.05) & (r < 0.1)] = float("-inf")
        s[(r >= 0.1) & (r < 0.13)] = float("nan")
        s[(r >= 0.13) & (r < 0.2)] = -0.0
        s[(r >= 0.2) & (r < 0.25)] = 0.0
        s[(r >= 0.25) & (r < 0.3)] = torch.finfo(torch.float32).min
    return s


def evict(scores, lens, retain, H, wide, slots, pad, option, max_len=None):
    from compactor_vllm import _native as N
    from compactor_vllm.compression.common import extract_and_store_top_kv

    n, B = sum(lens), len(lens)
    g = torch.Generator().manual_seed(5)
    k, v = (torch.randn(n, H, D, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    lens0 = torch.randint(0, 300, (B, H), generator=g).to(torch.int32).to(DEV)
    P = -(-(max(lens) + 300 + PS) // PS)
    rows = (B + 2) * H * P * PS
    table = torch.randperm((B + 2) * H * P, generator=g).to(torch.int32).view(B + 2, H, P).to(DEV)
    kc, vc = (torch.zeros(rows, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    buf = torch.zeros(n, H + (3 if wide else 0), device=DEV)
    buf[:, :H] = scores.to(DEV)
    cu = [0]
    for x in lens:
        cu.append(cu[-1] + x)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    N.set_test_option("select_passes", option)
    try:
        extract_and_store_top_kv(scores=buf[:, :H], cu_seqlens_k=i32(cu), max_k_len=max_len or max(lens), top_k=max(lens) * H, H=H,
                                 new_keys=k, new_vals=v, num_tokens_to_retain=i32(retain), page_table=table,
                                 batch_mapping=i32(slots), bh_lens=lens0, k_cache=kc, v_cache=vc, PAGE_SIZE=PS,
                                 PAD_TO_PAGE_SIZE=pad)
    finally:
        N.set_test_option("select_passes", 0)
    return lens0, kc, vc


LENS = {"one": [700], "ragged": [1, 2500, 0, 256, 257, 1023], "cluster2": [2600, 40], "cluster8": [15000, 3000, 7], "tiny": [3]}


@pytest.mark.parametrize("kind", ["random", "ties", "equal", "special"])
@pytest.mark.parametrize("lens", sorted(LENS))
@pytest.mark.parametrize("H", [1, 3, 8, 16])
def test_one_launch_equals_the_chain(H, lens, kind):
    L = LENS[lens]
    B = len(L)
    g = torch.Generator().manual_seed(H * 100 + B)
    scores = scores_of(kind, sum(L), H, g)
    slots = list(range(1, B + 1))
    if B > 3:
        slots[3] = 0                         # a reserved slot
    for ratio, pad, wide in ((0.5, True, False), (0.03, False, True), (1.0, True, False), (0.0, True, True)):
        retain = [int(round(ratio * x * H)) for x in L]
        if ratio == 0.03:
            retain = [max(1, r) for r in retain]
        a = evict(scores, L, retain, H, wide, slots, pad, 0)
        b = evict(scores, L, retain, H, wide, slots, pad, 1)
        for x, y in zip(a, b):
            assert torch.equal(x, y), (ratio, pad)


@pytest.mark.parametrize("n,H", [(40960, 8), (41216, 8), (16384, 16), (22000, 16)])
def test_where_the_clusters_end(n, H):
    """The largest sequences that a cluster's shared memory holds, and the first that it does not."""
    g = torch.Generator().manual_seed(n)
    scores = scores_of("random", n, H, g)
    a = evict(scores, [n], [n * H // 4], H, False, [1], True, 0)
    b = evict(scores, [n], [n * H // 4], H, False, [1], True, 1)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


def launches(scores, lens, H, **kw):
    from compactor_vllm import _native as N

    count = N.lib().cvllm_launch_count
    before = count()
    out = evict(scores, lens, [n * H // 2 for n in lens], H, False, list(range(1, len(lens) + 1)), True, 0, **kw)
    return count() - before, out


def test_the_longest_sequence_chooses_the_path():
    """Sequences that each fit a cluster take the two launches whatever their number; one that does not, the chain."""
    g = torch.Generator().manual_seed(3)
    for lens, want in (([6000] * 12, 2), ([40960, 300], 2), ([41216, 300], 13), ([200] * 300, 2)):
        scores = scores_of("random", sum(lens), 8, g)
        n, got = launches(scores, lens, 8)
        assert n == want, (lens[0], len(lens), n)
        chain = evict(scores, lens, [x * 4 for x in lens], 8, False, list(range(1, len(lens) + 1)), True, 1)
        for x, y in zip(got, chain):
            assert torch.equal(x, y)


@pytest.mark.parametrize("kind", ["random", "ties", "special"])
@pytest.mark.parametrize("H,bound", [(8, 1), (8, 300), (8, 5000), (3, 256), (16, 2049)])
def test_sequences_longer_than_the_bound(H, bound, kind):
    """max_k_len below the longest sequence: keys beyond a cluster's share are read where they are, with the same result."""
    lens = [700, 9001, 256, 0, 2300]
    g = torch.Generator().manual_seed(H + bound)
    scores = scores_of(kind, sum(lens), H, g)
    retain, slots = [n * H // 3 for n in lens], [1, 2, 3, 4, 5]
    a = evict(scores, lens, retain, H, True, slots, True, 0, max_len=bound)
    b = evict(scores, lens, retain, H, True, slots, True, 1)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("D", [8, 32, 64, 128, 256])
@pytest.mark.parametrize("H,lens,ratio", [(1, [1], 1.0), (16, [255, 257, 1], 0.5), (8, [3000, 512], 0.37), (3, [777] * 9, 0.9),
                                          (2, [160000, 300], 0.05), (8, [2048], 0.0005)])
def test_kept_rows_are_where_they_belong(D, H, lens, ratio):
    """Rows of 16 to 512 bytes, one to eight copy CTAs per tile: every head's kept tokens in ascending order, nothing else moved."""
    from compactor_vllm.compression.common import extract_and_store_top_kv

    B, PS, n = len(lens), 64, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(D + H)
    flat = torch.randn(n * H, generator=g, device=DEV)
    scores = flat.view(n, H)
    k, v = (torch.randn(n, H, D, generator=g, device=DEV).bfloat16() for _ in range(2))
    pages = max(lens) // PS + 2
    table = torch.randperm((B + 1) * H * pages, generator=g, device=DEV).to(torch.int32).view(B + 1, H, pages).contiguous()
    kc, vc = (torch.full((table.numel() * PS, D), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    want_k, want_v = kc.clone(), vc.clone()
    lens0 = torch.randint(0, 3, (B, H), generator=g, device=DEV).to(torch.int32)
    start, want_lens, cu, retain = lens0.clone(), lens0.clone(), [0], []
    for b, m in enumerate(lens):
        at, keep = cu[-1], int(ratio * m * H)
        cu.append(at + m)
        retain.append(keep)
        kept = torch.zeros(m * H, dtype=torch.bool, device=DEV)
        kept[flat[at * H:(at + m) * H].argsort(descending=True, stable=True)[:keep]] = True
        for h in range(H):
            tok = kept.view(m, H)[:, h].nonzero()[:, 0]
            pos = start[b, h] + torch.arange(tok.numel(), device=DEV)
            rows = table[b + 1, h, (pos // PS).long()].long() * PS + pos % PS
            want_k[rows], want_v[rows] = k[at + tok, h], v[at + tok, h]
            want_lens[b, h] += tok.numel()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    extract_and_store_top_kv(scores=scores, cu_seqlens_k=i32(cu), max_k_len=max(lens), top_k=max(lens) * H, H=H, new_keys=k,
                             new_vals=v, num_tokens_to_retain=i32(retain), page_table=table, batch_mapping=i32(list(range(1, B + 1))),
                             bh_lens=lens0, k_cache=kc, v_cache=vc, PAGE_SIZE=PS, PAD_TO_PAGE_SIZE=False)
    assert torch.equal(lens0, want_lens) and torch.equal(kc, want_k) and torch.equal(vc, want_v)

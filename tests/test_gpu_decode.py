"""Decode attention through head_sparse_decode_attention vs the CPU oracle / golden vectors."""
import pytest
import torch

from compactor_vllm.attention.sparse_decode_kernel import head_sparse_decode_attention
from oracle import attention as oa

from conftest import load_golden
from helpers import make_paged

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = {torch.float16: 3e-3, torch.bfloat16: 2e-2}  # reference test atol 3e-3 (fp16); 2e-2 bf16


def _check(q, kc, vc, lens, pt, bm, HKV, PS, dtype, scale=None):
    out = head_sparse_decode_attention(q, kc, vc, lens, pt, bm, HKV, PS, scale)
    torch.cuda.synchronize()
    ref = oa.decode_attention(q.cpu(), kc.cpu(), vc.cpu(), lens.cpu(), pt.cpu(), bm.cpu(), HKV, PS, scale)
    assert torch.isfinite(out).all()
    err = (out.float().cpu() - ref).abs().max().item()
    assert err <= TOL[dtype], err
    return out


@pytest.mark.parametrize("name", ["decode_bf16", "decode_f16"])
def test_decode_golden(name):
    g = load_golden(name)
    dtype = g["q"].dtype
    out = head_sparse_decode_attention(g["q"].to(DEV), g["k_cache"].to(DEV), g["v_cache"].to(DEV),
                                       g["seq_lens_bh"].to(DEV), g["page_table"].to(DEV),
                                       g["batch_mapping"].to(DEV), g["HKV"], g["PS"])
    valid = g["valid_rows"]
    err = (out.float().cpu()[valid] - g["out"].float()[valid]).abs().max().item()
    assert err <= TOL[dtype], err
    assert (out.float().cpu()[~valid] == 0).all()


# the reference's own grid: tests/test_triton_attention.py:52-68 (B x cache_len, HQ=32 HKV=8 D=128)
@pytest.mark.parametrize("B", [1, 2, 3, 8])
@pytest.mark.parametrize("cache_len", [1, 2, 70, 128, 8000])
def test_decode_reference_grid(B, cache_len):
    dtype, HQ, HKV, D, PS = torch.float16, 32, 8, 128, 256
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, [[cache_len] * HKV] * B, dtype, DEV, seed=1234)
    g = torch.Generator().manual_seed(B * 1000 + cache_len)
    q = torch.randn((B, HQ, D), generator=g).to(dtype).to(DEV)
    lens = torch.full((B, HKV), cache_len, dtype=torch.int32, device=DEV)
    _check(q, kc, vc, lens, pt, bm, HKV, PS, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("HQ,HKV,PS", [(32, 8, 128), (8, 1, 128), (16, 2, 32), (32, 8, 64)])
def test_decode_head_sparse_poisoned(dtype, HQ, HKV, PS):
    """Ragged per-head lengths, empty heads, scrambled pages, non-identity slots, NaN in every
    cache row a kernel has no business reading."""
    B, D = 5, 128
    g = torch.Generator().manual_seed(HQ + PS)
    lens = torch.randint(0, 3000, (B, HKV), generator=g)
    lens[0, 0] = 0
    lens[1, :] = 0
    lens[2, -1] = 1
    lens[3, 0] = 2048
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens.tolist(), dtype, DEV, seed=11, poison=True)
    q = torch.randn((B, HQ, D), generator=g).to(dtype).to(DEV)
    out = _check(q, kc, vc, lens.to(torch.int32).to(DEV), pt, bm, HKV, PS, dtype, scale=0.11)
    G = HQ // HKV
    empty = (lens == 0).repeat_interleave(G, dim=1)
    assert (out.cpu()[empty] == 0).all()


def test_decode_q_4d_and_key_split_independent():
    dtype, B, HQ, HKV, D, PS = torch.bfloat16, 2, 32, 8, 128, 128
    lens = [[5000] * HKV, [300] * HKV]
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens, dtype, DEV, seed=2)
    q = torch.randn((B, HQ, 1, D), generator=torch.Generator().manual_seed(0)).to(dtype).to(DEV)
    l = torch.tensor(lens, dtype=torch.int32, device=DEV)
    a = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS, None, key_split=1)
    b = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS, None, key_split=7)
    assert a.shape == (B, HQ, D)
    assert torch.equal(a, b)


def test_decode_large_batch_balanced():
    """Config-3-like raggedness at reduced size: many heads, many CTAs share heads."""
    dtype, B, HQ, HKV, D, PS = torch.bfloat16, 16, 32, 8, 128, 128
    g = torch.Generator().manual_seed(9)
    lens = torch.randint(1, 6000, (B, HKV), generator=g)
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens.tolist(), dtype, DEV, seed=5)
    q = torch.randn((B, HQ, D), generator=g).to(dtype).to(DEV)
    _check(q, kc, vc, lens.to(torch.int32).to(DEV), pt, bm, HKV, PS, dtype)


def test_decode_cuda_graph_capturable():
    dtype, B, HQ, HKV, D, PS = torch.bfloat16, 4, 32, 8, 128, 128
    lens = torch.randint(1, 2000, (B, HKV), generator=torch.Generator().manual_seed(1))
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens.tolist(), dtype, DEV, seed=8)
    q = torch.randn((B, HQ, D), generator=torch.Generator().manual_seed(2)).to(dtype).to(DEV)
    l = lens.to(torch.int32).to(DEV)
    eager = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)  # warm the workspace
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)
    torch.cuda.current_stream().wait_stream(s)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


def test_decode_step_matches_store_then_attend_with_reserved_rows():
    """cvllm_decode_step (slot-indexed lengths, what Attention.forward's decode branch calls) against the
    reference-shaped sequence index_select -> decode_store_kv -> attention -> index_copy_, bit for bit;
    rows mapped to RESERVED_BATCH (CUDA-graph padding, core/model_runner.py:484) are skipped."""
    from compactor_vllm.attention.sparse_decode_kernel import decode_append_and_attend
    from compactor_vllm.kv_cache.store_kv_cache import decode_store_kv
    dtype, B, HQ, HKV, D, PS = torch.bfloat16, 6, 32, 8, 128, 128
    g = torch.Generator().manual_seed(4)
    lens = torch.randint(0, 1500, (B, HKV), generator=g)
    lens[2, 3] = 0
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, (lens + 2).tolist(), dtype, DEV, seed=21, n_extra_slots=3)
    bm = bm.clone()
    bm[1] = 0
    bm[4] = 0  # two padding rows
    n_slots = pt.shape[0]
    table = torch.zeros((n_slots, HKV), dtype=torch.int32, device=DEV)
    table[bm.long()] = lens.to(torch.int32).to(DEV)
    table[0] = 0
    q = torch.randn((B, HQ, D), generator=g).to(dtype).to(DEV)
    kn = torch.randn((B, HKV, D), generator=g).to(dtype).to(DEV)
    vn = torch.randn((B, HKV, D), generator=g).to(dtype).to(DEV)

    kc2, vc2, table2 = kc.clone(), vc.clone(), table.clone()
    gathered = table2.index_select(0, bm.long()).contiguous()
    decode_store_kv(key=kn, value=vn, batch_mapping=bm, bh_lens=gathered, page_table=pt, k_cache=kc2,
                    v_cache=vc2, PAGE_SIZE=PS)
    ref = head_sparse_decode_attention(q, kc2, vc2, gathered, pt, bm, HKV, PS)
    live = bm != 0
    table2[bm[live].long()] = gathered[live]

    out = decode_append_and_attend(q, kn, vn, kc, vc, table, pt, bm, HKV, PS)
    torch.cuda.synchronize()
    assert torch.equal(table, table2) and (table[0] == 0).all()
    assert torch.equal(kc.view(torch.int16), kc2.view(torch.int16)) and torch.equal(vc.view(torch.int16), vc2.view(torch.int16))
    assert torch.equal(out[live], ref[live])
    assert (out[~live] == 0).all()


@pytest.mark.parametrize("HQ,HKV,PS", [(32, 8, 128), (8, 1, 64)])
@pytest.mark.parametrize("B,units", [(1, 4), (1, 5), (2, 8), (20, 6), (40, 7), (40, 8), (40, 9), (130, 5), (130, 6),
                                     (1, 20), (1, 147), (1, 148), (1, 149), (3, 49)])
def test_decode_whole_and_cut_heads(HQ, HKV, PS, B, units):
    """Both sides of the rule that leaves short heads whole (longest head 4, 5, 6, 8 units of 128 rows beside shares of under
    one, up to six and more than six units per CTA), and cut heads over fewer, as many and more units than CTAs, with empty heads, one-row heads and NaN behind every head's end."""
    dtype, D = torch.bfloat16, 128
    g = torch.Generator().manual_seed(100 * B + units)
    lens = torch.randint(1, units * 128 + 1, (B, HKV), generator=g)
    lens[torch.rand((B, HKV), generator=g) < 0.15] = 0
    lens[B // 2, 0], lens[0, -1] = 1, units * 128
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens.tolist(), dtype, DEV, seed=B + units, poison=True)
    q = torch.randn((B, HQ, D), generator=g).to(dtype).to(DEV)
    out = _check(q, kc, vc, lens.to(torch.int32).to(DEV), pt, bm, HKV, PS, dtype)
    assert (out.cpu()[(lens == 0).repeat_interleave(HQ // HKV, dim=1)] == 0).all()


@pytest.mark.parametrize("B,HQ,HKV", [
    (4499, 32, 8), (31319, 8, 1),      # the most sequences that the heads' prefix leaves two ring slots for
    (1600, 4, 1), (1900, 4, 1),        # the table of slot numbers beside six ring slots, and the first size where it would cost one
    (3700, 4, 1)])                     # five slots without it
def test_decode_many_sequences(B, HQ, HKV):
    dtype, D, PS, pages = torch.bfloat16, 128, 32, 64
    g = torch.Generator(device=DEV).manual_seed(B)
    kc, vc = (torch.randn(pages * PS, D, generator=g, device=DEV).to(dtype) for _ in range(2))
    pt = torch.randint(0, pages, (B + 1, HKV, 2), generator=g, device=DEV, dtype=torch.int32)
    lens = torch.randint(0, 2 * PS + 1, (B, HKV), generator=g, device=DEV, dtype=torch.int32)
    bm = (torch.randperm(B, generator=g, device=DEV) + 1).to(torch.int32)
    q = torch.randn(B, HQ, D, generator=g, device=DEV).to(dtype)
    out = head_sparse_decode_attention(q, kc, vc, lens, pt, bm, HKV, PS, 0.1)
    for b0 in range(0, B, 1024):
        s = slice(b0, b0 + 1024)
        at = (pt[bm[s].long()].long()[..., None] * PS + torch.arange(PS, device=DEV)).flatten(-2)       # [b, HKV, 2 PS]
        k, v = kc.float()[at], vc.float()[at]
        x = torch.einsum("bhgd,bhnd->bhgn", q[s].float().view(-1, HKV, HQ // HKV, D), k) * 0.1
        there = torch.arange(2 * PS, device=DEV) < lens[s][:, :, None]
        x = x.masked_fill(~there[:, :, None], -torch.inf).softmax(-1).nan_to_num(0.0)
        want = torch.einsum("bhgn,bhnd->bhgd", x, v).flatten(1, 2)
        assert (out[s].float() - want).abs().max().item() <= TOL[dtype]


@pytest.mark.parametrize("captured", [False, True])
def test_decode_behind_another_stream(captured):
    """The launch is scheduled beside the kernel in front of it: what it reads may come from another stream that was waited for just
    before, or from a copy in front, and what follows may overwrite its inputs."""
    dtype, B, HQ, HKV, D, PS = torch.bfloat16, 4, 32, 8, 128, 128
    lens = torch.randint(1, 3000, (B, HKV), generator=torch.Generator().manual_seed(5))
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens.tolist(), dtype, DEV, seed=9)
    g = torch.Generator(device=DEV).manual_seed(6)
    q = torch.randn((B, HQ, D), generator=g, device=DEV).to(dtype)
    l = lens.to(torch.int32).to(DEV)
    want = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)
    q_now, l_now, big = torch.zeros_like(q), torch.zeros_like(l), torch.randn((1 << 24,), device=DEV)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def step():
        side.wait_stream(main)
        with torch.cuda.stream(side):
            for _ in range(4):
                big.mul_(1.0)               # the copies come late
            q_now.copy_(q)
            l_now.copy_(l)
        first = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)
        main.wait_stream(side)
        second = head_sparse_decode_attention(q_now, kc, vc, l_now, pt, bm, HKV, PS)
        third = head_sparse_decode_attention(second.clone().copy_(q_now), kc, vc, l_now, pt, bm, HKV, PS)
        q_now.zero_()
        l_now.zero_()
        return first, second, third

    with torch.cuda.stream(main):
        outs = step()
        if captured:
            main.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=main):
                outs = step()
            for o in outs:
                o.zero_()
            for _ in range(3):
                graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("HQ,HKV,rows", [(32, 8, 384), (16, 8, 130), (8, 1, 384), (32, 8, 6000)])     # whole heads; cut ones
def test_decode_infinite_values(HQ, HKV, rows, dtype):
    """An infinite value that a query sees makes its number infinite, not NaN, and leaves the others as they are."""
    B, D, PS = 6, 128, 128
    lens = torch.randint(rows // 2, rows + 1, (B, HKV), generator=torch.Generator().manual_seed(rows))
    kc, vc, pt, bm = make_paged(B, HKV, D, PS, lens.tolist(), dtype, DEV, seed=rows)
    g = torch.Generator(device=DEV).manual_seed(7)
    q = (0.1 * torch.randn((B, HQ, D), generator=g, device=DEV)).to(dtype)
    l = lens.to(torch.int32).to(DEV)
    want = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)
    first = pt[bm.long(), :, 0].long().flatten() * PS
    vc[first + 5, 3], vc[first + 9, 4] = torch.inf, -torch.inf
    out = head_sparse_decode_attention(q, kc, vc, l, pt, bm, HKV, PS)
    assert (out[..., 3] == torch.inf).all() and (out[..., 4] == -torch.inf).all()
    rest = torch.arange(D, device=DEV).sub(3.5).abs() > 1
    assert torch.equal(out[..., rest], want[..., rest])

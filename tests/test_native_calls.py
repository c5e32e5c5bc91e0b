"""The calls that take tensors (csrc/host/py_call.cpp) against the long way: same results, same refusals."""
import ctypes

import numpy as np
import pytest
import torch

from compactor_vllm import _native as N
from compactor_vllm.attention.sparse_decode_kernel import head_sparse_decode_attention
from compactor_vllm.attention.sparse_varlen_kernel import causal_sparse_varlen_with_cache

DEV = "cuda"


def test_host_tensors_are_refused():
    L, t = N.lib(), torch.zeros(4, 8, 128, dtype=torch.float16)
    assert L.call.bind("no such function", 1, None) is None
    assert L.call.decode_attention(L.decode_address, {}, t, t, t, t, t, t, 8, 128, None) is None
    assert L.call.prefill_attention(L.prefill_address, *[t] * 9, 1, 1, 8, 128, None) is None
    with pytest.raises(AssertionError, match="CUDA tensors"):
        L.cvllm_decode_attention(t, *[None] * 7, 0, 1, 32, 8, 128, 128, 1, 0.1, 0, 0, None)


def test_other_arguments_go_to_ctypes():
    L = N.lib()
    count = (ctypes.c_int * 1)()
    # B = 0: nothing is launched; a ctypes array among the arguments, and a call with an argument too many
    args = [None, count, *[None] * 6, 0, 0, 32, 8, 128, 128, 1, 0.1, 0, 0, None]
    assert L.cvllm_decode_attention(*args) == 0
    assert L.cvllm_decode_attention(*[None] * 8, 0, 0, 32, 8, 128, 128, 1, 1, 0, True, None) == 0
    with pytest.raises(TypeError):
        L.cvllm_decode_attention(1, 2)
    with pytest.raises(ctypes.ArgumentError):
        L.cvllm_decode_attention(*[None] * 8, 0, "one", 32, 8, 128, 128, 1, 0.1, 0, 0, None)


class Placed(torch.Tensor):
    """Says of itself that it lies on a GPU, at an address."""
    is_cuda = True

    def data_ptr(self):
        return 4096


@pytest.mark.parametrize("number", [np.int64, np.int32, torch.tensor], ids=["int64", "int32", "tensor"])
def test_numbers_of_other_libraries_beside_tensors(number):
    """ctypes takes what has an __index__ or a __float__ where the ABI has a number; beside it the tensors still pass as addresses."""
    L, t = N.lib(), torch.zeros(1).as_subclass(Placed)
    scale = np.float32(0.1) if number is not torch.tensor else torch.tensor(0.1)
    rest = [number(x) for x in (8, 128, 128, 1)]
    # B = 0: nothing is launched
    assert L.cvllm_decode_attention(*[t] * 8, number(0), number(0), number(32), *rest, scale, number(0), number(0), None) == 0
    with pytest.raises(AssertionError, match="CUDA tensors"):
        L.cvllm_decode_attention(*[t] * 7, torch.zeros(1), 0, number(0), 32, 8, 128, 128, 1, 0.1, 0, 0, None)
    seen = []
    bound = L.call.bind("cvllm_decode_attention", 1, lambda *a: seen.append(a) or 5)
    assert bound(*[t] * 7, None, 0, number(0), 32, 8, 128, 128, 1, 0.1, 0, 0, None) == 5
    assert seen[0][:8] == (4096,) * 7 + (None,) and seen[0][10:] == (32, 8, 128, 128, 1, 0.1, 0, 0, None)
    assert bound(t, t) == 5 and seen[1] == (4096, 4096)
    assert bound(*[0] * 19, t) == 5 and seen[2][19] is t


class Named(torch.Tensor):
    pass


def _long_way(monkeypatch):
    class Never:
        decode_attention = prefill_attention = staticmethod(lambda *a: None)

    lib = N.lib()
    other = type(lib)(**vars(lib))
    other.call = Never
    monkeypatch.setattr(N, "lib", lambda: other)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["plain", "default scale", "int64", "four dims", "strided lengths", "subclass", "int scale"])
def test_decode_forms(monkeypatch, form, dtype):
    B, HQ, HKV, PS, pages = 3, 16, 4, 32, 9
    g = torch.Generator(device=DEV).manual_seed(3)
    q = torch.randn(B, HQ, 128, generator=g, device=DEV).to(dtype)
    kc, vc = (torch.randn((B + 1) * HKV * pages * PS, 128, generator=g, device=DEV).to(dtype) for _ in range(2))
    pt = torch.randperm((B + 1) * HKV * pages, generator=g, device=DEV).to(torch.int32).view(B + 1, HKV, pages).contiguous()
    lens = torch.randint(1, pages * PS, (B, HKV), generator=g, device=DEV).to(torch.int32)
    bm, scale = torch.tensor([2, 1, 3], dtype=torch.int32, device=DEV), 0.07
    if form == "default scale":
        scale = None
    elif form == "int64":
        lens = lens.long()
    elif form == "four dims":
        q = q[:, :, None]
    elif form == "strided lengths":
        lens = lens.t().contiguous().t()
    elif form == "subclass":
        q, lens = q.as_subclass(Named), lens.as_subclass(Named)
    elif form == "int scale":
        scale = 1
    run = lambda: head_sparse_decode_attention(q, kc, vc, lens, pt, bm, HKV, PS, scale)  # noqa: E731
    run()                                     # the workspace
    got, L = run(), N.lib()
    short = L.call.decode_attention(L.decode_address, N._WORKSPACES, q, kc, vc, lens, pt, bm, HKV, PS, scale)
    assert torch.equal(short, got) if form in ("plain", "default scale") else short is None
    with pytest.raises(AssertionError):
        head_sparse_decode_attention(q, kc, vc, lens, pt[:, :2].contiguous(), bm, HKV, PS, scale)
    with pytest.raises(AssertionError):
        head_sparse_decode_attention(q, kc, vc, lens, pt, bm.long(), HKV, PS, scale)
    _long_way(monkeypatch)
    assert torch.equal(got, run()) and got.shape == (B, HQ, 128)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "views", "default scale", "int64", "no bound", "bound of 64 bits", "subclass"])
def test_prefill_forms(monkeypatch, form):
    lens, HQ, HKV, PS, pages = [5, 130, 64], 8, 2, 128, 4
    B, n, dtype = len(lens), sum(lens), torch.bfloat16
    g = torch.Generator(device=DEV).manual_seed(4)
    rows = torch.randn(n, HQ + 2 * HKV, 128, generator=g, device=DEV).to(dtype)
    q, k, v = rows[:, :HQ], rows[:, HQ:HQ + HKV], rows[:, HQ + HKV:]
    if form != "views":
        q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    kc, vc = (torch.randn((B + 1) * HKV * pages * PS, 128, generator=g, device=DEV).to(dtype) for _ in range(2))
    pt = torch.randperm((B + 1) * HKV * pages, generator=g, device=DEV).to(torch.int32).view(B + 1, HKV, pages).contiguous()
    past = torch.randint(0, pages * PS, (B, HKV), generator=g, device=DEV).to(torch.int32)
    cu = torch.tensor([0, 5, 135, 199], dtype=torch.int32, device=DEV)
    bm, scale, bound = torch.tensor([2, 1, 3], dtype=torch.int32, device=DEV), 0.07, pages * PS
    if form == "default scale":
        scale = None
    elif form == "int64":
        cu, past, bm = cu.long(), past.long(), bm.long()
    elif form == "no bound":
        bound = None
    elif form == "bound of 64 bits":
        bound = 1 << 40
    elif form == "subclass":
        q = q.as_subclass(Named)
    call = lambda q=q, k=k, pt=pt: causal_sparse_varlen_with_cache(  # noqa: E731
        q, k, v, kc, vc, seq_lens_bh=past, global_page_table=pt, batch_mapping=bm, cu_seqlens_q=cu, max_seqlen_q=130,
        max_seqlen_k_cache=bound, HKV=HKV, PAGE_SIZE=PS, sm_scale=scale)
    got, L = call(), N.lib()
    short = L.call.prefill_attention(L.prefill_address, q, k, v, kc, vc, past, pt, bm, cu, 130, bound, HKV, PS, scale)
    served = ("plain", "views", "default scale", "bound of 64 bits")
    assert torch.equal(short, got) if form in served else short is None
    with pytest.raises(AssertionError):
        call(k=k[:-1])
    with pytest.raises(AssertionError):
        call(q=q.half())
    with pytest.raises(AssertionError):
        call(pt=pt.long())
    _long_way(monkeypatch)
    assert torch.equal(got, call()) and got.shape == (n, HQ, 128)


@pytest.mark.gpu
@pytest.mark.parametrize("transform", ["vmap", "grad", "jvp", "vmap of lengths"])
def test_tensors_without_memory_are_refused(transform):
    """Inside vmap and the transforms of torch.func a tensor is of the exact type and contiguous, but has no address: an exception as
    for every call that asks for one, and the next call works."""
    B, HQ, HKV, PS, pages = 2, 8, 2, 128, 1
    g = torch.Generator(device=DEV).manual_seed(5)
    q = torch.randn(B, HQ, 128, generator=g, device=DEV, dtype=torch.bfloat16)
    kc, vc = (torch.randn((B + 1) * HKV * pages * PS, 128, generator=g, device=DEV).to(q.dtype) for _ in range(2))
    k, v = (torch.randn(B, HKV, 128, generator=g, device=DEV).to(q.dtype) for _ in range(2))
    pt = torch.randperm((B + 1) * HKV * pages, generator=g, device=DEV).to(torch.int32).view(B + 1, HKV, pages).contiguous()
    lens = torch.full((B, HKV), 40, dtype=torch.int32, device=DEV)
    bm, cu = torch.tensor([2, 1], dtype=torch.int32, device=DEV), torch.arange(B + 1, dtype=torch.int32, device=DEV)

    def decode(q, lens=lens):
        return head_sparse_decode_attention(q, kc, vc, lens, pt, bm, HKV, PS, 0.1)

    def prefill(q, lens=lens):
        return causal_sparse_varlen_with_cache(q, k, v, kc, vc, seq_lens_bh=lens, global_page_table=pt, batch_mapping=bm,
                                               cu_seqlens_q=cu, max_seqlen_q=1, max_seqlen_k_cache=40, HKV=HKV, PAGE_SIZE=PS,
                                               sm_scale=0.1)

    for attend in (decode, prefill):
        want = attend(q)                        # and the workspace
        with pytest.raises(RuntimeError, match="Cannot access data pointer"):
            if transform == "vmap":
                torch.vmap(attend)(q[None].expand(3, -1, -1, -1).contiguous())
            elif transform == "grad":
                torch.func.grad(lambda x: attend(x).float().sum())(q)
            elif transform == "jvp":
                torch.func.jvp(attend, (q,), (q,))
            else:
                torch.vmap(lambda x: attend(q, x))(lens[None].expand(3, -1, -1).contiguous())
        assert torch.equal(attend(q), want)

"""Norm, rotation and store of heads with one and with four tokens per CTA (csrc/bias_attn.cu): groups of four that the tokens do not
fill, that cross sequences and hold tokens of the reserved slot, value sizes other than the key's, both types, and the cache
lengths, which above 64 tokens the last token of an ascending run raises alone.

Both must give the same bits; against 64 bits: 32-bit sums of up to 128 squares and a rotation, 1e-5; bfloat16 rows are rounded
once, 2^-9 of the value, and near zero the rotation's cancellation counts, 2^-9 of the row's largest."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rot", [0, 32])
@pytest.mark.parametrize("size", [(4, 2, 64, 64), (3, 1, 128, 96), (2, 2, 32, 48), (8, 4, 128, 128)], ids=str)
@pytest.mark.parametrize("T", [1, 3, 66, 67, 130])
def test_one_and_four_tokens(T, size, rot, dtype):
    from compactor_vllm import _native as N

    H, G, D, Dv = size
    eps, ps, pages = 1e-5, 8, 30
    g = torch.Generator().manual_seed(T + D)
    qkv = torch.randn(T, (H + G) * D + G * Dv, generator=g).to(dtype)
    # slots 1 .. 3 in runs of three, the reserved slot 0 among them; positions of a slot ascend, jump back and repeat
    slots = [(t // 3) % 4 for t in range(T)]
    rank, positions = [0, 0, 0, 0], []
    for s in slots:
        positions.append(100 - rank[s] if s == 2 and rank[s] % 5 == 4 else rank[s])
        rank[s] += 1
    if T > 20:      # the same token twice: equal rows, so that it does not matter which is stored last
        slots[17], positions[17], qkv[17] = slots[16], positions[16], qkv[16]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, slot, rows = i32(positions), i32(slots), qkv.to(DEV)
    wq, wk = (1 + 0.2 * torch.randn(2, D, generator=g)).to(DEV)
    freq = torch.rand(rot // 2, generator=g).double().to(DEV) if rot else None
    order = torch.randperm(4 * G * pages, generator=g)
    table = order.to(torch.int32).view(4, G, pages).to(DEV)

    def run(tokens):
        q = torch.empty(T, H, D, dtype=dtype, device=DEV)
        kc, vc = torch.zeros(4 * G * pages * ps, D, dtype=dtype, device=DEV), torch.zeros(4 * G * pages * ps, Dv, dtype=dtype, device=DEV)
        lens = torch.zeros(4, G, dtype=torch.int32, device=DEV)
        N.set_test_option("qknorm_tokens", tokens)
        try:
            N.check(N.lib().cvllm_rope_qknorm_store(
                N.ptr(rows), rows.stride(0), N.ptr(freq), rot, 3, N.ptr(wq), N.ptr(wk), eps, N.ptr(pos), N.ptr(slot), N.ptr(q),
                N.ptr(kc), N.ptr(vc), N.ptr(table), table.stride(0), table.stride(1), ps, N.ptr(lens), T, H, G, D, Dv, 0,
                N.block_dtype_code(dtype), N.stream(q.device)), "store")
        finally:
            N.set_test_option("qknorm_tokens", 0)
        return q, kc, vc, lens

    one, four = run(1), run(4)
    for x, y in zip(one, four):
        assert torch.equal(x, y)
    q, kc, vc, lens = (x.cpu() for x in four)
    want_lens = [0 if s == 0 else max([p + 1 for p, o in zip(positions, slots) if o == s], default=0) for s in range(4)]
    assert lens.tolist() == [[n] * G for n in want_lens]

    def rotated(x):
        x = x.clone()
        if rot:
            a = torch.tensor(positions).double()[:, None, None] * freq.cpu()
            u, v = x[..., 0:rot:2].clone(), x[..., 1:rot:2].clone()
            x[..., 0:rot:2], x[..., 1:rot:2] = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
        return x

    x = qkv.double()
    want_q = unit(rotated(x[:, :H * D].view(T, H, D)), eps) * wq.cpu().double()
    want_k = unit(rotated(x[:, H * D:(H + G) * D].view(T, G, D)), eps) * wk.cpu().double()
    want_v = unit(x[:, (H + G) * D:].view(T, G, Dv), eps)
    near = 1e-5 if dtype == torch.float32 else 2 ** -8
    close = lambda got, want: torch.allclose(got.double(), want, rtol=near, atol=near)
    assert close(q, want_q)
    stored = torch.zeros(kc.shape[0], dtype=torch.bool)
    for t in range(T):
        if slots[t] == 0:
            continue
        for h in range(G):
            row = int(order.view(4, G, pages)[slots[t], h, positions[t] // ps]) * ps + positions[t] % ps
            stored[row] = True
            assert close(kc[row], want_k[t, h]) and close(vc[row], want_v[t, h])
    assert not kc[~stored].any() and not vc[~stored].any()

"""The gated delta rule's kernels over the layouts that they choose from (key sizes that leave rows of the state tile empty,
value columns over clusters of CTAs, two and four columns per thread, stages and blocks that portions do not fill), against
the recurrence token by token in 64 bits.

Tolerance: everything behind the inputs is 32-bit; a state entry sums up to a few hundred products of unit vectors, decayed, so
sqrt(300) * 2^-24 = 1e-6 relative; 1e-5 leaves the coefficients' triangular solve its own rounding.  bfloat16 rows are rounded
at the output only: 2^-9 / sqrt(3) = 1.1e-3, and 2.5e-3 is twice that."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def setup(heads, kv, dim, vdim, lens, starts, dtype, seed):
    from compactor_vllm.layers.recurrent import DeltaRuleMixer

    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)
    m = DeltaRuleMixer(heads * vdim, heads, kv, dim, vdim, 3, 1e-6).to(DEV)
    with torch.no_grad():
        m.conv_weight.copy_(0.6 * r(*m.conv_weight.shape))
        m.A_log.copy_(r(heads) - 1.0)
        m.dt_bias.copy_(r(heads) - 2.0)
        m.norm_weight.copy_(1.0 + 0.1 * r(vdim))
    m.requires_grad_(False)
    m.o_proj = torch.nn.Identity()
    state = m.make_state()
    for name, (shape, kind) in state.state_specs(dtype).items():
        setattr(state, name, (0.3 * r(len(lens) + 1, *shape)).to(kind))
    cols = r(sum(lens), m.in_cols).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ctx = dict(is_prefill=max(lens) > 1, cu_seqlens_q=i32(cu), max_seqlen_q=max(lens),
               batch_mapping=i32(list(range(1, len(lens) + 1))), seq_start=i32(starts), positions_i32=i32(starts))
    return m, state, cols, ctx


def recurrence(m, state, cols, lens, starts):
    H, G, D, Dv = m.heads, m.kv_heads, m.dim, m.vdim
    S_all, out, at, C = state.matrix_state.double().clone(), [], 0, m.conv_channels
    for b, (n, start) in enumerate(zip(lens, starts)):
        x = cols[at:at + n].double()
        before = state.conv_state[b + 1].double() if start else torch.zeros(m.taps - 1, C, dtype=torch.float64, device=DEV)
        raw = torch.cat([before, x[:, :C]])
        y = sum(raw[t:t + n] * m.conv_weight[:, t].double() for t in range(m.taps))
        y = y * torch.sigmoid(y)
        unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
        q = (unit(y[:, :G * D].view(n, G, D)) * D ** -0.5).repeat_interleave(H // G, 1)
        k = unit(y[:, G * D:2 * G * D].view(n, G, D)).repeat_interleave(H // G, 1)
        v = y[:, 2 * G * D:].view(n, H, Dv)
        gate, beta = x[:, C:C + H * Dv], torch.sigmoid(x[:, C + H * Dv:C + H * Dv + H])
        decay = torch.exp(-torch.exp(m.A_log.double()) *
                          torch.nn.functional.softplus(x[:, C + H * Dv + H:] + m.dt_bias.double(), threshold=100.0))
        S = S_all[b + 1] if start else torch.zeros_like(S_all[b + 1])
        o = torch.empty(n, H, Dv, dtype=torch.float64, device=DEV)
        for t in range(n):
            S = S * decay[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None]
            o[t] = torch.einsum("hvk,hk->hv", S, q[t])
        S_all[b + 1] = S
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * m.norm_weight.double()
        out.append(o.reshape(n, H * Dv) * gate * torch.sigmoid(gate))
        at += n
    return torch.cat(out), S_all


SIZES = [(2, 1, 128, 128), (4, 2, 64, 64), (3, 3, 20, 12), (2, 2, 7, 5), (1, 1, 256, 256), (2, 1, 130, 34), (2, 1, 40, 200),
         (2, 1, 6, 256)]
LENS = [([97], [0]), ([1, 4, 33, 130], [5, 0, 9, 0]), ([2], [0]), ([64, 3], [3, 0])]


@pytest.mark.parametrize("layout", [0, 102, 104, 202, 404, 802])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_portions(size, layout):
    run(size, LENS, layout, torch.float32)


@pytest.mark.parametrize("size", SIZES, ids=str)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_single_tokens_and_types(size, dtype):
    run(size, [([1], [0]), ([1, 1, 1], [4, 0, 77])] + LENS[:2], 0, dtype)


def run(size, lens, layout, dtype):
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context, set_context

    for n, (ls, starts) in enumerate(lens):
        m, state, cols, ctx = setup(*size, ls, starts, dtype, 3 + n)
        want, want_state = recurrence(m, state, cols, ls, starts)
        untouched = state.matrix_state[0].clone()
        set_context(**ctx)
        N.set_test_option("gla_layout", layout)
        try:
            got = m(None, cols, state).double()
        finally:
            N.set_test_option("gla_layout", 0)
            reset_context()
        err = lambda x, y: ((x - y).norm() / y.norm()).item()
        assert err(got, want) < (1e-5 if dtype == torch.float32 else 2.5e-3), (ls, err(got, want))
        assert err(state.matrix_state[1:].double(), want_state[1:]) < 1e-5, ls
        assert torch.equal(state.matrix_state[0], untouched)
        assert math.isfinite(got.sum().item())


@pytest.mark.parametrize("layout", [0, 102, 104, 404])
@pytest.mark.parametrize("at", [1, 6, 7, 34, 63])
def test_what_is_not_finite_stays_behind_its_token(at, layout):
    """An infinite or NaN entry of one token's row changes no bit of the tokens before it or of other sequences, whatever
    place of its block the token has."""
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context, set_context

    heads, kv, dim, vdim = 2, 1, 64, 64
    lens, starts = [70, 9], [3, 0]
    channels = 2 * kv * dim + heads * vdim
    # a query, a key, a value, the gate, beta and the decay
    places = [3, kv * dim + 5, 2 * kv * dim + 7, channels + 2, channels + heads * vdim, channels + heads * vdim + heads]

    def once(place, value):
        m, state, cols, ctx = setup(heads, kv, dim, vdim, lens, starts, torch.float32, 21)
        if place is not None:
            cols[at, place] = value
        set_context(**ctx)
        N.set_test_option("gla_layout", layout)
        try:
            return m(None, cols, state), state.matrix_state
        finally:
            N.set_test_option("gla_layout", 0)
            reset_context()

    clean, clean_state = once(None, None)
    assert torch.isfinite(clean).all()
    for place in places:
        for value in (math.inf, -math.inf, math.nan):
            got, state = once(place, value)
            assert torch.equal(got[:at], clean[:at]) and torch.equal(got[lens[0]:], clean[lens[0]:]), (place, value)
            assert torch.equal(state[2], clean_state[2])
            assert value == value or not torch.isfinite(got[at:lens[0]]).all()

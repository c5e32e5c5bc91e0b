"""The gated delta rule's portions in chunks of 64 tokens (one tile of the tensor cores), against the recurrence token by token
in 64 bits: chunks that are full, one token short and one token long, heads that share keys, clusters of one to eight CTAs,
both types, and portions whose images exceed the workspace's bound and are taken in windows; the convolution in front with
its rows in four-channel pieces and without.

Tolerances: operands in three bfloat16 parts are good to 2^-26, coefficients are 64-bit, the tensor pipe's sums of 64 and 128
products fp32.  Measured over the sizes here 1.2e-7 to 3.5e-7 in 32-bit outputs and states; the bound is about twice that, where
a build without the third parts lies at 4e-6 and above.  bfloat16 rows are rounded at the output only: 2^-9 / sqrt(3) = 1.1e-3,
and 2.5e-3 is twice that."""
import ctypes

import pytest
import torch

import test_gpu_delta_layouts as layouts
from test_gpu_delta_layouts import recurrence, setup

pytestmark = pytest.mark.gpu


def check(size, lens, starts, dtype, seed=5, odd_rows=False):
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context, set_context

    m, state, cols, ctx = setup(*size, lens, starts, dtype, seed)
    N.set_test_option("gla_layout", -1)       # chunks whatever the length
    # rows on 16 bytes, or a view whose rows do not start there: the kernels of the shorter portions
    wide = torch.zeros(cols.shape[0], (cols.shape[1] + 8) // 8 * 8, dtype=dtype, device=cols.device)
    at = 1 if odd_rows else 0
    wide[:, at:at + cols.shape[1]] = cols
    cols = wide[:, at:at + cols.shape[1]]
    if odd_rows:
        assert cols.data_ptr() % 16 != 0
    else:
        heads, kv, dim, vdim = size
        assert N.lib().cvllm_delta_rule_chunks_workspace_bytes(sum(lens), len(lens), max(lens), heads, kv, dim, vdim) > 0
    want, want_state = recurrence(m, state, cols, lens, starts)
    untouched, before = state.matrix_state[0].clone(), aborts()
    set_context(**ctx)
    launched = N.lib().cvllm_launch_count()
    try:
        got = m(None, cols, state).double()
    finally:
        N.set_test_option("gla_layout", 0)
        reset_context()
    # the convolution, its state, then one kernel, or three per window of chunks
    launched = N.lib().cvllm_launch_count() - launched - 2
    assert launched == 1 if odd_rows else launched >= 3 and launched % 3 == 0
    assert aborts() == before
    err = lambda x, y: ((x - y).norm() / y.norm()).item()
    near = 1e-5 if odd_rows else 7e-7       # the blocks of four: test_gpu_delta_layouts.py
    assert err(got, want) < (near if dtype == torch.float32 else 2.5e-3), err(got, want)
    assert err(state.matrix_state[1:].double(), want_state[1:]) < near, err(state.matrix_state[1:].double(), want_state[1:])
    assert torch.equal(state.matrix_state[0], untouched)
    return launched


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens, starts", [([64], [0]), ([65, 1, 128, 63], [7, 0, 0, 3]), ([127, 200], [0, 9])])
@pytest.mark.parametrize("size", [(2, 1, 128, 128), (4, 2, 64, 64), (3, 1, 128, 32), (2, 2, 64, 96), (1, 1, 128, 256)], ids=str)
def test_chunks(size, lens, starts, dtype):
    check(size, lens, starts, dtype)


def shared_direction(kind, m, cols, seed):
    """Keys that share a direction, as a convolution with silu leaves them: a drift under noise, one key for all tokens, one
    token repeated, and keys of alternating sign with beta and decays near 1."""
    draw = torch.Generator().manual_seed(seed)
    r = lambda n: torch.randn(n, generator=draw).to(cols.device)
    qk, values, C = 2 * m.kv_heads * m.dim, m.heads * m.vdim, m.conv_channels
    if kind == "drift":
        cols[:, :qk] = 0.5 * cols[:, :qk] + 1.5 * r(qk)
    elif kind == "one key":
        cols[:, :qk] = r(qk)
    elif kind == "one token":
        cols[:, :C] = r(C)
    elif kind == "alternating":
        sign = torch.ones(cols.shape[0], 1, device=cols.device)
        sign[::2] = -1
        cols[:, :qk] = sign * 4 * r(qk) + 0.01 * cols[:, :qk]
        cols[:, C + values:C + values + m.heads] = 6.0 + 0.1 * cols[:, C + values:C + values + m.heads]
        m.A_log.fill_(-6.0)


@pytest.mark.parametrize("size", [(4, 2, 128, 128), (4, 2, 64, 64)], ids=str)
@pytest.mark.parametrize("lens", [[1000], [128], [130, 70, 333]], ids=str)
@pytest.mark.parametrize("kind", ["random", "drift", "one key", "one token", "alternating"])
def test_no_farther_from_64_bits_than_the_blocks_of_four(kind, lens, size):
    """Root mean square over six draws of both kernels' distances from 64 bits, 32-bit rows, outputs and states.  The chunks lie
    at 0.3 to 0.9 of the blocks of four; with 32-bit coefficients, or all of K S in one accumulator, at up to 2.4."""
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context, set_context

    square = {-1: [0.0, 0.0], 102: [0.0, 0.0]}
    for seed in range(3, 9):
        for layout, sums in square.items():
            m, state, cols, ctx = setup(*size, lens, [0] * len(lens), torch.float32, seed)
            shared_direction(kind, m, cols, seed + 100)
            want, want_state = recurrence(m, state, cols, lens, [0] * len(lens))
            set_context(**ctx)
            N.set_test_option("gla_layout", layout)
            try:
                got = m(None, cols, state).double()
            finally:
                N.set_test_option("gla_layout", 0)
                reset_context()
            for i, (x, y) in enumerate([(got, want), (state.matrix_state[1:].double(), want_state[1:])]):
                sums[i] += ((x - y).norm() / y.norm()).item() ** 2
    for chunks, blocks in zip(square[-1], square[102]):
        assert chunks <= blocks, ((chunks / 6) ** 0.5, (blocks / 6) ** 0.5)


def test_rows_off_the_grid():
    check((2, 1, 128, 128), [130, 70], [0, 4], torch.float32, odd_rows=True)


@pytest.mark.parametrize("at", [1, 15, 16, 34, 63, 64, 69])
def test_what_is_not_finite_stays_behind_its_token(at):
    layouts.test_what_is_not_finite_stays_behind_its_token(at, -1)


def test_the_rule():
    """Short portions, batches of mostly short ones and, for few value columns, many (head, sequence) pairs are the other
    kernel's."""
    from compactor_vllm import _native as N

    def need(lens, heads, dim, vdim):
        return N.lib().cvllm_delta_rule_chunks_workspace_bytes(sum(lens), len(lens), max(lens), heads, heads // 2, dim, vdim) > 0

    assert need([192], 16, 128, 128) and not need([191], 16, 128, 128)
    assert need([128] * 5, 16, 128, 128) and not need([128] * 4, 16, 128, 128) and not need([127] * 8, 16, 128, 128)
    assert need([959, 1], 16, 128, 128) and not need([959] + [1] * 10, 16, 128, 128)
    assert need([384], 32, 64, 256) and not need([383], 32, 64, 256) and need([256] * 2, 32, 64, 256) and need([128] * 9, 32, 64, 256)
    assert need([256], 16, 128, 64) and need([512] * 2, 32, 128, 64) and not need([511] * 2, 32, 128, 64)
    assert not need([4096] * 3, 32, 64, 64) and need([512] * 3, 16, 128, 32) and not need([4096] * 4, 16, 128, 32)


def aborts():
    from compactor_vllm import _native as N

    count = ctypes.c_int(-1)
    N.check(N.lib().cvllm_delta_chunk_aborts(ctypes.byref(count)), "aborts")
    return count.value


@pytest.mark.parametrize("lens", [[200, 64], [192]], ids=str)
@pytest.mark.parametrize("hold", [1, 2, 3, -1, -2, -3])
@pytest.mark.parametrize("vdim", [32, 64])
def test_a_wait_that_runs_out(vdim, hold, lens):
    """Copies that never begin (a flag that nothing sets): the call ends, the counter goes up, what the affected CTAs would have
    written is NaN - rows and state of head 0, the cluster's other columns too, which wait for its sums - and the other heads' work
    is what it was."""
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context, set_context

    def once(held):
        m, state, cols, ctx = setup(2, 1, 64, vdim, lens, [0] * len(lens), torch.float32, 11)
        set_context(**ctx)
        N.set_test_option("gla_layout", -1)
        N.set_test_option("delta_chunk_hold", held)
        try:
            out = m(None, cols, state)
        finally:
            N.set_test_option("delta_chunk_hold", 0)
            N.set_test_option("gla_layout", 0)
            reset_context()
        return out.view(-1, 2, vdim), state.matrix_state

    before = aborts()
    clean, clean_state = once(0)
    assert aborts() == before and torch.isfinite(clean).all() and torch.isfinite(clean_state).all()
    got, state = once(hold)
    assert aborts() > before
    at = 0
    for b, n in enumerate(lens):
        if n > 64 * (abs(hold) - 1):
            first = 0 if hold > 0 else 64 * (-hold - 1)        # a chunk kernel's rows are void, a coefficient's from its chunk on
            assert torch.isnan(got[at + first:at + n, 0]).all() and torch.isnan(state[b + 1, 0]).all()
            assert torch.equal(got[at:at + first, 0], clean[at:at + first, 0])
        else:
            assert torch.equal(got[at:at + n, 0], clean[at:at + n, 0]) and torch.equal(state[b + 1, 0], clean_state[b + 1, 0])
        at += n
    assert torch.equal(got[:, 1], clean[:, 1]) and torch.equal(state[1:, 1], clean_state[1:, 1])


@pytest.mark.parametrize("size, lens, windows", [
    ((32, 32, 128, 128), [7000, 300], 3), ((32, 32, 128, 128), [1, 2500, 64, 1, 3000, 127, 900], 3),
    ((32, 16, 128, 128), [6000] + [1] * 31, 2), ((2, 1, 64, 64), [1] * 300 + [130, 70], 1),
    ((8, 8, 128, 64), [3300, 3200, 3100, 3000], 2)], ids=["two", "seven", "one long", "many", "about equal"])
def test_windows(size, lens, windows):
    """Chunks of all sequences in one row, cut into windows of 320 MB: what a window holds does not depend on how the tokens are
    spread over the sequences.  The last: a range of every sequence's chunks, for few heads and sequences about equally long."""
    starts = [11 * (i % 2) for i in range(len(lens))]
    assert check(size, lens, starts, torch.bfloat16) == 3 * windows


def test_without_memory_for_the_images(monkeypatch):
    """A device that has no room left for the workspace: the kernel that needs none, as before there were chunks."""
    from compactor_vllm import _native as N
    from compactor_vllm.utils.context import reset_context, set_context

    m, state, cols, ctx = setup(4, 2, 128, 128, [400], [0], torch.float32, 6)
    want, want_state = recurrence(m, state, cols, [400], [0])
    empty = torch.empty

    def full(*args, **kw):
        if kw.get("dtype") is torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", full)
    set_context(**ctx)
    launched = N.lib().cvllm_launch_count()
    try:
        got = m(None, cols, state)
    finally:
        reset_context()
    assert N.lib().cvllm_launch_count() - launched == 3
    for x, y in ((got, want), (state.matrix_state[1:], want_state[1:])):
        assert ((x.double() - y).norm() / y.norm()).item() < 1e-5


def test_silu_without_a_division():
    """The convolution's rows in four-channel pieces make their silu from an approximate reciprocal and a correction, rows off the
    16-byte grid by a division: the same bits over the whole range, where the denominator's reciprocal is subnormal too, and for
    infinities and NaN."""
    from compactor_vllm import _native as N

    C, T, dev = 4096, 256, "cuda"
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    x = torch.linspace(-104.0, 104.0, T * C, device=dev)[torch.randperm(T * C, generator=torch.Generator().manual_seed(1)).to(dev)].view(T, C)
    x[:, :256] = torch.linspace(-88.8, -87.2, T * 256, device=dev).view(T, 256)
    x[-3] = 0.0          # what follows a number that is not finite is NaN: its weight is 0
    x[-2] = torch.tensor([float("inf"), -float("inf"), float("nan"), 3e38, -3e38, 1e-40, -1e-40, -0.0], device=dev).repeat(C // 8)
    weight = torch.zeros(C, 2, device=dev)
    weight[:, 1] = 1.0
    state, cu, zero, slot = torch.zeros(2, 1, C, device=dev), i32([0, T]), i32([0]), i32([1])

    def silu(off):
        rows = torch.zeros(T, C + 4, device=dev)
        rows[:, off:off + C] = x
        out = torch.empty(T, C, device=dev)
        N.check(N.lib().cvllm_causal_conv(N.ptr(rows), rows.stride(0), off, C, 2, N.ptr(weight), None, N.ptr(state), N.ptr(cu),
                                          N.ptr(zero), None, N.ptr(slot), 1, T, N.ptr(out), C, N.block_dtype_code(x.dtype),
                                          N.stream(out.device)), "cvllm_causal_conv")
        return out

    got, want = silu(0), silu(1)
    assert torch.equal(got.nan_to_num(nan=7.0), want.nan_to_num(nan=7.0)) and torch.equal(got.isnan(), want.isnan())
    assert torch.equal(torch.signbit(got[:-1]), torch.signbit(want[:-1]))
    exact = x[:-3].double() * torch.sigmoid(x[:-3].double())
    # expf is good to 2^-22, the sum and the quotient to 2^-24 each; below 1e-30 e^-z nears the end of fp32's range
    normal = exact.abs() > 1e-30
    assert ((got[:-3].double() - exact)[normal].abs() <= (2 ** -22 + 2 ** -23) * exact[normal].abs()).all()

"""The gated delta rule by chunks of 16 tokens: against the recurrence in float64, outputs and the whole state behind them, on
portions around whole chunks, several entries a step, states that are not zero, tokens that continue a portion (carried
convolution inputs), grouped heads, values of other sizes, fewer taps, decays that underflow and decays of nearly one."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DK, EPS = 128, 1e-6


class Ctx:
    dtype = torch.bfloat16

    def __init__(self, lens, slots):
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        self.cu_q, self.slots, self.n_entries, self.max_q_len = i32(cu), i32(slots), len(lens), max(lens)
        self.entry_of_token = i32([e for e, n in enumerate(lens) for _ in range(n)])
        self.host = {"q_lens": lens}
        from safetyraise_lmengine_b200.parts.base import Workspace
        self.workspace = Workspace(torch.device(DEV), cu[-1])


def recurrence(proj, conv_w, a_log, dt_bias, state, H, G, dv, taps, eps=EPS):
    """One entry in float64 -> (o [n, H, dv], the state row behind it)."""
    n, C = proj.shape[0], 2 * G * DK + H * dv
    S = state[:H * DK * dv].view(H, dv, DK).transpose(1, 2).clone()
    carry = state[H * DK * dv:].view(C, taps - 1).T
    x = torch.cat([carry, proj[:, :C]])
    y = sum(x[j:j + n] * conv_w[:, j] for j in range(taps))
    y = y * torch.sigmoid(y)
    unit = lambda a: a / torch.sqrt((a * a).sum(-1, keepdim=True) + eps)
    q, k = unit(y[:, :G * DK].view(n, G, DK)) * DK ** -0.5, unit(y[:, G * DK:2 * G * DK].view(n, G, DK))
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    v = y[:, 2 * G * DK:].view(n, H, dv)
    beta = torch.sigmoid(proj[:, C:C + H])
    g = torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(proj[:, C + H:C + 2 * H] + dt_bias))
    o = torch.empty(n, H, dv, dtype=torch.float64, device=proj.device)
    for t in range(n):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        o[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return o, torch.cat([S.transpose(1, 2).reshape(-1), x[n:].T.reshape(-1)])


@pytest.mark.parametrize("H, G, dv, taps", [(2, 2, 128, 4), (4, 2, 48, 4), (3, 1, 16, 2), (2, 1, 144, 1), (1, 1, 128, 3)])
@pytest.mark.parametrize("lens", [[16], [1, 17, 2, 33], [15, 31, 48], [130]])
@pytest.mark.parametrize("eps", [EPS, 0.0])                  # 0: the places behind an entry's last token have no length
def test_against_float64(H, G, dv, taps, lens, eps):
    from safetyraise_lmengine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H + dv + taps + len(lens))
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    C, T = 2 * G * DK + H * dv, sum(lens)
    row = H * DK * dv + C * (taps - 1)
    row += row % 2
    state = rand(6, row)
    slots = [4, 1, 5, 2][:len(lens)]
    proj = rand(T, C + 2 * H + H * dv + 3)
    proj[T // 2:, C + H:C + 2 * H] += 8.0            # decays that underflow within a chunk, behind decays of nearly one
    conv_w, dt_bias = rand(C, taps) * 0.5, rand(H) - 4.0
    a_log = torch.log(1.0 + 15.0 * torch.rand(H, generator=gen, device=DEV))
    before = state.double().clone()
    ctx = Ctx(lens, slots)
    o = torch.empty(T, H * dv, device=DEV)
    n = ops.delta_by_chunks(ctx, state, DK, dv, taps)
    if max(lens) < ops.DELTA_CHUNKS_FROM:
        assert n == 0
        return
    assert n == sum(-(-x // 16) for x in lens if x >= ops.DELTA_CHUNKS_FROM)
    ops.delta_chunks(ctx, proj, conv_w, a_log, dt_bias, state, o, n, H, G, DK, dv, taps, eps)
    want_o, want_state, t = [], before.clone(), 0
    for x, slot in zip(lens, slots):
        used = H * DK * dv + C * (taps - 1)
        a, b = recurrence(proj[t:t + x].double(), conv_w.double(), a_log.double(), dt_bias.double(), before[slot, :used], H, G, dv, taps, eps)
        want_o.append(a.reshape(x, -1))
        want_state[slot, :used] = b
        t += x
    want_o = torch.cat(want_o)
    # float32 sums over 128 rows and 16 tokens of terms of about one: a few hundred roundings of 2^-24
    assert (o.double() - want_o).abs().max() <= 2e-5 * want_o.abs().max()
    assert (state.double() - want_state).abs().max() <= 2e-5 * want_state.abs().max()
    untouched = [s for s in range(6) if s not in slots]
    assert torch.equal(state[untouched].double(), before[untouched])


@pytest.mark.parametrize("lens", [[16], [100], [33, 300], [700]])
def test_no_further_from_float64_than_token_by_token(lens):
    """Step sizes between 0.001 and 0.1 and rates up to 16, spread over their logarithm, as models are initialised."""
    from safetyraise_lmengine_b200.kernels import ops
    H, dv, taps, T = 16, 128, 4, sum(lens)
    C = 3 * H * DK
    gen = torch.Generator(device=DEV).manual_seed(T)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    uniform = lambda lo, hi: lo + (hi - lo) * torch.rand(H, generator=gen, device=DEV)
    proj, conv_w, a_log = 0.9 * rand(T, C + 2 * H + H * dv), 0.4 * rand(C, taps), torch.log(uniform(1.0, 16.0))
    step = torch.exp(uniform(math.log(1e-3), math.log(1e-1)))
    dt_bias = step + torch.log(-torch.expm1(-step))
    start = torch.zeros(len(lens), H * DK * dv + C * (taps - 1), device=DEV)
    ctx, used = Ctx(lens, list(range(len(lens)))), H * DK * dv
    want_o, want_s, t = [], [], 0
    for e, n in enumerate(lens):
        a, b = recurrence(proj[t:t + n].double(), conv_w.double(), a_log.double(), dt_bias.double(), start[e].double(), H, H, dv, taps)
        want_o.append(a.reshape(n, -1))
        want_s.append(b[:used])
        t += n
    want_o, want_s = torch.cat(want_o), torch.stack(want_s)
    rel = lambda x, y: float((x.double() - y).norm() / y.norm())
    state, o = start.clone(), torch.empty(T, H * dv, device=DEV)
    qkv, beta, decay, qk = (torch.empty(T, n, device=DEV) for n in (C, H, H, H))
    ops.delta_prepare(ctx, proj, conv_w, a_log, dt_bias, state, qkv, beta, decay, qk, H, H, DK, dv, taps, EPS)
    ops.delta_recurrence(ctx, qkv, beta, decay, qk, state, o, H, H, DK, dv)
    walk = rel(o, want_o), rel(state[:, :used], want_s)
    state, o = start.clone(), torch.empty(T, H * dv, device=DEV)
    ops.delta_chunks(ctx, proj, conv_w, a_log, dt_bias, state, o, ops.delta_by_chunks(ctx, state, DK, dv, taps), H, H, DK, dv, taps, EPS)
    chunks = rel(o, want_o), rel(state[:, :used], want_s)
    # sums over 1e5 numbers and more: an error of this kind repeats itself within a few hundredths from seed to seed
    assert chunks[0] <= 1.05 * walk[0] and chunks[1] <= 1.05 * walk[1], (chunks, walk)


def test_the_float32_path_and_short_steps_go_token_by_token():
    from safetyraise_lmengine_b200.kernels import ops
    state = torch.zeros(1, 128 * 128 + 3 * 384, device=DEV)
    ctx = Ctx([64], [0])
    assert ops.delta_by_chunks(ctx, state, 128, 128, 4) == 4
    ctx.dtype = torch.float32
    assert ops.delta_by_chunks(ctx, state, 128, 128, 4) == 0
    assert ops.delta_by_chunks(Ctx([15, 4], [0, 0]), state, 128, 128, 4) == 0
    assert ops.delta_by_chunks(Ctx([64], [0]), state, 64, 128, 4) == 0
    assert ops.delta_by_chunks(Ctx([64], [0]), state[:, 1:], 128, 128, 4) == 0


def walked(lens, held=None, max_tokens=None):
    """(o, state, the workspace's generation) of a step of these entries, four heads of 128, inputs that depend on the entry alone."""
    from safetyraise_lmengine_b200.kernels import ops
    H, dv, taps = 4, 128, 4
    C = 3 * H * DK
    parts, states = [], []
    for e, n in enumerate(lens):
        g = torch.Generator(device=DEV).manual_seed(100 + e)
        states.append(torch.randn(H * DK * dv + C * (taps - 1), generator=g, device=DEV))
        parts.append(torch.randn(n, C + 2 * H + H * dv, generator=g, device=DEV))
    g = torch.Generator(device=DEV).manual_seed(7)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)
    conv_w, dt_bias, a_log = rand(C, taps) * 0.5, rand(H) - 4.0, rand(H)
    ctx, state = Ctx(lens, list(range(len(lens)))), torch.stack(states)
    if max_tokens:
        ctx.workspace.max_tokens = max_tokens
    o = torch.full((sum(lens), H * dv), float("nan"), device=DEV)
    was = type(ops).DELTA_CHUNKS_HELD
    try:
        type(ops).DELTA_CHUNKS_HELD = held or was
        n = ops.delta_by_chunks(ctx, state, DK, dv, taps)
        ops.delta_chunks(ctx, torch.cat(parts), conv_w, a_log, dt_bias, state, o, n, H, H, DK, dv, taps, EPS)
    finally:
        type(ops).DELTA_CHUNKS_HELD = was
    return o, state, ctx.workspace


@pytest.mark.parametrize("held", [1, 3, 5, 8])
def test_steps_whose_chunks_are_taken_by_turns(held):
    """Records for fewer chunks than a step has: the same bits, whatever lies together."""
    lens = [70, 16, 33, 100]
    o, state, _ = walked(lens)
    o2, state2, work = walked(lens, held)
    assert torch.equal(o, o2) and torch.equal(state, state2)
    assert max(b.shape[0] for (name, _, _), b in work._bufs.items() if name == "delta.records") == 4 * held


@pytest.mark.parametrize("lens", [[16, 40, 40, 100, 17], [100, 1, 16, 16, 300, 3, 16], [17, 1, 20] * 85, [17, 1, 20, 33] * 64, [20, 1, 17] * 86])
def test_entries_in_the_order_of_their_length(lens):
    """Equal lengths, short ones between them, as many entries as a block has threads (256) and more: the blocks take the longest
    first, and every entry's bits are those of a step of the first few alone."""
    o, state, _ = walked(lens)
    for first in (1, 5):
        alone, alone_state, _ = walked(lens[:first])
        assert torch.equal(o[:sum(lens[:first])].isnan(), alone.isnan())
        long = [t for t, n in zip(torch.arange(sum(lens[:first])).split(lens[:first]), lens) if n >= 16]
        rows = torch.cat(long).to(DEV)
        assert torch.equal(o[rows], alone[rows]) and torch.equal(state[:first], alone_state)


def test_an_entry_does_not_depend_on_who_shares_the_step():
    """A decoded token, a few tokens and a portion: the same bits beside others and alone (the walk, or the chunks)."""
    from safetyraise_lmengine_b200.kernels import ops
    lens, H, dv, taps = [1, 40, 3, 15, 16], 4, 128, 4
    C = 3 * H * DK
    g = torch.Generator(device=DEV).manual_seed(11)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, states = rand(sum(lens), C + 2 * H + H * dv), rand(len(lens), H * DK * dv + C * (taps - 1))
    conv_w, dt_bias, a_log = rand(C, taps) * 0.5, rand(H) - 4.0, rand(H)

    def go(lens, slots, rows):
        ctx, state = Ctx(lens, slots), states.clone()
        o = torch.full((sum(lens), H * dv), float("nan"), device=DEV)
        n = ops.delta_by_chunks(ctx, state, DK, dv, taps)
        if n:
            ops.delta_chunks(ctx, rows, conv_w, a_log, dt_bias, state, o, n, H, H, DK, dv, taps, EPS)
        else:
            ops.delta_walk(ctx, rows, conv_w, a_log, dt_bias, state, o, H, H, DK, dv, taps, EPS)
        return o, state

    o, state = go(lens, list(range(len(lens))), proj)
    t = 0
    for e, n in enumerate(lens):
        alone_o, alone_state = go([n], [e], proj[t:t + n].contiguous())
        assert torch.equal(alone_o, o[t:t + n]) and torch.equal(alone_state[e], state[e])
        t += n


def test_the_records_do_not_grow_with_the_portions():
    """Portions of growing length leave the workspace where it is: a buffer that moves throws the recorded decode graphs away."""
    from safetyraise_lmengine_b200.kernels import ops
    H, dv, taps, most = 2, 128, 4, 4096
    C = 3 * H * DK
    work = None
    for lens in ([16], [17] * 8, [400], [1000, 40], [4096], [17] * 240):
        ctx = Ctx(lens, list(range(len(lens))))
        work = ctx.workspace = work or type(ctx.workspace)(torch.device(DEV), most)
        state = torch.zeros(len(lens), H * DK * dv + C * (taps - 1), device=DEV)
        T = sum(lens)
        ops.delta_chunks(ctx, torch.zeros(T, C + 2 * H + H * dv, device=DEV), torch.zeros(C, taps, device=DEV), torch.zeros(H, device=DEV),
                         torch.zeros(H, device=DEV), state, torch.empty(T, H * dv, device=DEV),
                         ops.delta_by_chunks(ctx, state, DK, dv, taps), H, H, DK, dv, taps, EPS)
        assert work.generation == 0
    assert sum(b.numel() * b.element_size() for (name, _, _), b in work._bufs.items() if name == "delta.records") <= 160 * H * 42000

"""Kernels that copy several neighbouring numbers at once where sizes and addresses allow it: bit for bit the results of the
same call on operands that do not allow it, at the edges of their tiles."""
import pytest
import torch

from safetyraise_lmengine_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _shifted(t):
    """The same numbers at an address that is no multiple of 16 bytes."""
    buf = torch.empty(1 + t.numel(), dtype=t.dtype, device=t.device)
    return buf[1:].view(t.shape).copy_(t)


class _Entries:
    def __init__(self, lens):
        self.n_entries, self.max_q_len = len(lens), max(lens)
        ends = torch.tensor(lens).cumsum(0).tolist()
        self.cu_q = torch.tensor([0] + ends, dtype=torch.int32, device=DEV)
        self.slots = torch.tensor(list(range(len(lens)))[::-1], dtype=torch.int32, device=DEV)
        self.entry_of_token = torch.tensor(sum(([e] * n for e, n in enumerate(lens)), []), dtype=torch.int32, device=DEV)


# (1,600 channels and three entries: more blocks than the form for two blocks an SM takes)
@pytest.mark.parametrize("channels,N", [(4, 4), (20, 8), (36, 12), (16, 16), (48, 20), (16, 64), (20, 128), (1600, 16), (1600, 4)])
@pytest.mark.parametrize("lens", [(1,), (15, 16, 17), (40, 100, 7), (33, 1, 160), (2, 530)])
def test_scan_and_its_convolution(channels, N, lens):
    g = torch.Generator().manual_seed(channels + N)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    ctx, T, taps = _Entries(lens), sum(lens), 4
    xz, dbc, dt = rnd(T, 2 * channels), rnd(T, 4 + 2 * N), rnd(T, channels)
    A, D, bias = -torch.rand(channels, N, generator=g).to(DEV), rnd(channels), rnd(channels)
    conv_w, conv_b, start = rnd(channels, taps), rnd(channels), rnd(len(lens), channels * (N + taps - 1))
    got = []
    for move in (lambda t: t, _shifted):
        state, inputs = start.clone(), move(xz)
        x, x_low = torch.empty(T, channels, device=DEV), torch.empty(T, channels, dtype=torch.bfloat16, device=DEV)
        ops.scan_conv(ctx, inputs, conv_w, conv_b, state, x, x_low, channels, N, taps)
        out = torch.empty(T, channels, dtype=torch.bfloat16, device=DEV)
        ops.selective_scan(ctx, x, inputs, move(dbc), 4, dt, bias, A, D, state, out, channels, N, taps)
        got.append((x, x_low, out, state))
    assert all(torch.isfinite(t).all() for t in got[0])
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("channels,N", [(16, 16), (20, 36), (16, 64), (20, 100), (20, 128)])
@pytest.mark.parametrize("lens", [(1,), (1, 5, 64), (3, 70)])
def test_states_of_the_scan_at_any_address(channels, N, lens):
    """Pairs of states and decays by one access each, and number by number where an address or the slots' stride forbids it."""
    g = torch.Generator().manual_seed(channels + N)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    ctx, T, taps = _Entries(lens), sum(lens), 4
    x, xz, dbc, dt = rnd(T, channels), rnd(T, 2 * channels), rnd(T, 4 + 2 * N), rnd(T, channels)
    A, D, bias = -torch.rand(channels, N, generator=g).to(DEV), rnd(channels), rnd(channels)
    size = channels * (N + taps - 1)
    start = rnd(len(lens), size)
    got = []
    for a, state in ((A, start.clone()), (_shifted(A), start.clone()), (A, _shifted(start)), (A, torch.full((len(lens), size + 1), 7.0, device=DEV))):
        state[:, :size] = start
        out = torch.empty(T, channels, device=DEV)
        ops.selective_scan(ctx, x, xz, dbc, 4, dt, bias, a, D, state, out, channels, N, taps)
        assert (state[:, size:] == 7.0).all()
        got.append((out, state[:, :size]))
    assert torch.isfinite(got[0][0]).all()
    for other in got[1:]:
        assert all(torch.equal(p, q) for p, q in zip(got[0], other))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [4, 508, 1020, 1024, 4100])
@pytest.mark.parametrize("add", [False, True])
def test_embedding_rows(dtype, H, add):
    g = torch.Generator().manual_seed(H)
    table, first = torch.randn(9, H, generator=g).to(DEV, dtype), torch.randn(5, H, generator=g).to(DEV)
    ids = torch.tensor([8, 0, 9, -1, 3], dtype=torch.int32, device=DEV)         # two outside the table
    bad, out = torch.zeros(1, dtype=torch.int32, device=DEV), first.clone()
    ops.embed_gather(ids, table, out, bad, scale=0.3, add=add)
    rows = table.float()[ids.long().clamp(0, 8)] * torch.tensor(0.3, device=DEV)
    rows[2:4] = 0
    assert int(bad) == 1
    # with add one rounding more may be folded away (a fused multiply-add): half a unit of the product
    tol = 2.0 ** -24 * rows.abs() if add else torch.zeros_like(rows)
    want = first + rows if add else rows
    assert ((out - want).abs() <= tol + (2.0 ** -23 * want.abs() if add else 0)).all()


@pytest.mark.parametrize("proj,act", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("T,H,dv", [(1, 1, 1), (3, 3, 33), (2, 5, 64), (3, 2, 65), (9, 4, 128), (2, 3, 200), (1, 2, 256), (2, 2, 300)])
@pytest.mark.parametrize("logistic", [False, True])
def test_gated_norm_of_the_delta_rule(proj, act, T, H, dv, logistic):
    g = torch.Generator().manual_seed(dv)
    o, w = torch.randn(T, H * dv, generator=g), torch.randn(dv, generator=g)
    p = torch.randn(T, 7 + H * dv, generator=g).to(proj)
    out = torch.empty(T, H * dv, dtype=act, device=DEV)
    ops.delta_output(o.to(DEV), w.to(DEV), 1e-6, p.to(DEV), 7, out, H, dv, logistic)
    x, z = o.double().view(T, H, dv), p[:, 7:].double().view(T, H, dv)
    want = x / (x.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double() * torch.sigmoid(z) * (1 if logistic else z)
    # dv + 8 float32 roundings of factors of the result, then the one of the output's own type
    tol = (dv + 8) * 2.0 ** -24 + (0 if act == torch.float32 else 2.0 ** -8)
    assert ((out.cpu().double().view(T, H, dv) - want).abs() <= tol * want.abs() + 1e-30).all()

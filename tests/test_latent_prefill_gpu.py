"""Prompts of a latent attention on the tensor-memory kernel: rows and keys at the edges of its tiles, pages of every form it
takes, windows with pages given back, both pairings of the rotation, the gate, operands whose rows are no whole 16-byte
pieces, and neighbours that must not be read."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DIM, ROT, DV, RANK = 128, 64, 128, 40


class Ctx:
    def __init__(self, q_lens, kv_lens):
        starts = [k - q for q, k in zip(q_lens, kv_lens)]
        cu = [0]
        for q in q_lens:
            cu.append(cu[-1] + q)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        self.cu_q, self.kv_lens, self.tables = i32(cu), i32(kv_lens), {}
        self.host = {"q_lens": q_lens, "kv_lens": kv_lens, "starts": starts}


@pytest.mark.parametrize("page", [8, 16, 64, 256])
@pytest.mark.parametrize("window", [0, 70, 300])
@pytest.mark.parametrize("heads, pairs, interleaved, gated", [(2, 32, True, True), (2, 32, False, False), (3, 16, False, False), (1, 0, True, True),
                                                               (2, 6, True, False)])
def test_prompts_against_float64(page, window, heads, pairs, interleaved, gated):
    from safetyraise_lmengine_b200.kernels import ops
    from safetyraise_lmengine_b200.parts.base import Rotation
    g = torch.Generator().manual_seed(page + window + heads)
    q_lens, kv_lens = [1, 128, 5, 257, 130], [1, 128, 300, 384, 515]
    T, scale = sum(q_lens), 0.5 * (DIM + ROT) ** -0.5
    ctx = Ctx(q_lens, kv_lens)
    wide = heads * (DIM + ROT) + (4 if heads == 2 else 1) + heads + heads % 2    # the gate's columns, behind the queries'
    q = torch.randn(T, wide, generator=g)
    first = [max(0, k - n - window + 1) if window else 0 for n, k in zip(q_lens, kv_lens)]
    cu_kv, keys = [], 0
    for f, k in zip(first, kv_lens):
        cu_kv.append(keys - f)
        keys += k - f
    rows = torch.randn(keys, heads * (DIM + DV), generator=g).bfloat16()
    n_pages = sum(-(-k // page) for k in kv_lens)
    order = torch.randperm(n_pages, generator=g).tolist()
    pages = torch.full((n_pages, 1, page, RANK + ROT), float("nan"), dtype=torch.bfloat16)
    shared = [torch.randn(k, ROT, generator=g).bfloat16() for k in kv_lens]
    table = torch.zeros(len(kv_lens), max(-(-k // page) for k in kv_lens) + 1, dtype=torch.int32)
    at = 0
    for e, k in enumerate(kv_lens):
        for b in range(-(-k // page)):
            if (b + 1) * page <= first[e]:
                table[e, b] = -1                                                 # behind the window: given back
                continue
            table[e, b] = order[at]
            lo, hi = b * page, min((b + 1) * page, k)
            pages[order[at], 0, :hi - lo, RANK:] = shared[e][lo:hi]
            at += 1
    cos = sin = rotation = None
    if pairs:
        angle = torch.randn(T, pairs, generator=g)
        cos, sin = angle.cos(), angle.sin()
        rotation = Rotation(cos.to(DEV), sin.to(DEV), pairs, interleaved)
    # the reference: queries rounded to bfloat16 once turned, as the kernel's operands are
    x = q[:, :heads * (DIM + ROT)].reshape(T, heads, DIM + ROT).clone()
    if pairs:
        c, s, tail = cos[:, None], sin[:, None], x[..., DIM:DIM + 2 * pairs].clone()
        a, b = (tail[..., 0::2], tail[..., 1::2]) if interleaved else (tail[..., :pairs], tail[..., pairs:])
        turned = (a * c - b * s, b * c + a * s)
        x[..., DIM:DIM + 2 * pairs] = torch.stack(turned, -1).flatten(-2) if interleaved else torch.cat(turned, -1)
    x = x.bfloat16().double()
    ref = torch.zeros(T, heads, DV, dtype=torch.float64)
    t = 0
    for e, (n, k) in enumerate(zip(q_lens, kv_lens)):
        mine = rows[cu_kv[e] + first[e]:cu_kv[e] + k].double()
        j = torch.arange(first[e], k)
        i = torch.arange(k - n, k)[:, None]
        seen = (j <= i) & (j > i - window if window else j >= 0)
        for h in range(heads):
            key = torch.cat([mine[:, h * DIM:(h + 1) * DIM], shared[e][first[e]:].double()], -1)
            p = torch.softmax((x[t:t + n, h] @ key.T * scale).masked_fill(~seen, -math.inf), -1)
            ref[t:t + n, h] = p @ mine[:, heads * DIM + h * DV:heads * DIM + (h + 1) * DV]
        t += n
    gate = None
    if gated:
        gate = (q.to(DEV), wide - heads)
        ref *= torch.sigmoid(q[:, -heads:].double())[:, :, None]
    out = torch.full((T, heads * DV), 7.0, dtype=torch.bfloat16, device=DEV)
    assert ops.latent_prefill_tcgen05_takes(q.to(DEV), DIM, ROT, DV, RANK, page)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.bind_error_flag(flag)
    try:
        ops.latent_prefill_tcgen05(ctx, q.to(DEV), rotation, pages.to(DEV), rows.to(DEV), torch.tensor(cu_kv, dtype=torch.int32, device=DEV),
                                   out, table.to(DEV), heads, DIM, ROT, DV, RANK, heads * DIM, scale, window, gate=gate)
        got = out.double().cpu().view(T, heads, DV)
    finally:
        ops.bind_error_flag(None)
    assert int(flag) == 0
    # weights and the result are rounded to 8 bits of mantissa (2^-9 each way): a value is a mean of N(0, 1) values under weights
    # that are off by 2^-9 of themselves, then off by 2^-9 of itself
    assert (got - ref).abs().max() <= 2.0 ** -8 * (1.0 + ref.abs().max())


def test_a_weight_that_outweighs_the_others_loses_nothing():
    """One key of every head has nearly all the weight and comes behind one that is e^4 to e^5.5 smaller: the output is its value
    but for what the other key adds, rounded once.  A weight rounded to 8 bits beside a sum that is not, or measured from a
    maximum that lags, would be off by up to 2^-8 of itself."""
    from safetyraise_lmengine_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    heads, n, k, page = 8, 130, 400, 16
    ctx = Ctx([n], [k])
    q = torch.zeros(n, heads * (DIM + ROT))
    q[:, ::DIM + ROT] = 1.0
    rows = torch.randn(k, heads * (DIM + DV), generator=g).bfloat16()
    rows[:, :heads * DIM:DIM] = -100.0
    rows[5, :heads * DIM:DIM] = 0.0
    rows[200, :heads * DIM:DIM] = (4.0 + 1.5 * torch.rand(heads, generator=g)).bfloat16()
    pages = torch.zeros(k // page, 1, page, RANK + ROT, dtype=torch.bfloat16, device=DEV)
    table = torch.arange(k // page, dtype=torch.int32, device=DEV)[None]
    out = torch.empty(n, heads * DV, dtype=torch.bfloat16, device=DEV)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.bind_error_flag(flag)
    try:
        ops.latent_prefill_tcgen05(ctx, q.to(DEV), None, pages, rows.to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV), out, table,
                                   heads, DIM, ROT, DV, RANK, heads * DIM, 1.0)
        got = out.double().cpu().view(n, heads, DV)
    finally:
        ops.bind_error_flag(None)
    assert int(flag) == 0
    small = torch.exp(-rows[200, :heads * DIM:DIM].double())[:, None]
    v = rows[:, heads * DIM:].double().view(k, heads, DV)
    ref = (v[200] + small * v[5]) / (1 + small)
    # half a step of the result's 8 bits, and 2^-8 of the small weight's part
    half = 2.0 ** (torch.floor(torch.log2(ref.abs())) - 8)
    assert ((got - ref).abs() <= half * 1.001 + 2.0 ** -8 * small * (v[5] - v[200]).abs() + 1e-6).all()


# (3 heads in blocks of 32 columns; 40 heads of 130 or 516 columns and up in the wide form, 148 blocks of 32 and more)
@pytest.mark.parametrize("heads", [3, 40])
@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 40])
@pytest.mark.parametrize("dim, rot, rank, dv", [(128, 64, 512, 128), (12, 6, 20, 9), (64, 0, 130, 33), (3, 2, 5, 1), (30, 4, 516, 132)])
@pytest.mark.parametrize("wdt", [torch.bfloat16, torch.float32])
def test_the_per_head_products(heads, T, dim, rot, rank, dv, wdt):
    """The up projections folded into the queries and applied behind the attention: token tiles of 8 and 16, sizes that are no
    whole pieces, columns beyond a block's 32; a token's result does not depend on its neighbours."""
    from safetyraise_lmengine_b200.kernels import ops
    g = torch.Generator().manual_seed(T + dim)
    q = torch.randn(T, heads * (dim + rot) + heads, generator=g)
    uk, uv = torch.randn(heads, dim, rank, generator=g).to(wdt), torch.randn(heads, rank, dv, generator=g).to(wdt)
    out = torch.empty(T, heads * (rank + rot), device=DEV)
    ops.latent_absorb(q.to(DEV), uk.to(DEV), None, out, heads, dim, rot, rank)
    x = q[:, :heads * (dim + rot)].view(T, heads, dim + rot).double()
    ref = torch.cat([torch.einsum("thd,hdr->thr", x[..., :dim], uk.double()), x[..., dim:]], -1)
    assert (out.cpu().double().view(ref.shape) - ref).abs().max() <= 1e-5 * ref.abs().max()
    o = torch.randn(T, heads * rank, generator=g)
    got = torch.empty(T, heads * dv, device=DEV)
    ops.latent_expand(o.to(DEV), uv.to(DEV), q.to(DEV), heads * (dim + rot), got, heads, rank, dv)
    ref = torch.einsum("thr,hrc->thc", o.view(T, heads, rank).double(), uv.double()) * torch.sigmoid(q[:, -heads:].double())[:, :, None]
    assert (got.cpu().double().view(ref.shape) - ref).abs().max() <= 1e-5 * ref.abs().max()
    one = torch.empty(1, heads * dv, device=DEV)
    ops.latent_expand(o[T - 1:].contiguous().to(DEV), uv.to(DEV), q[T - 1:].contiguous().to(DEV), heads * (dim + rot), one, heads, rank, dv)
    assert torch.equal(one[0], got[T - 1])
    folded = torch.empty(1, heads * (rank + rot), device=DEV)
    ops.latent_absorb(q[T - 1:].contiguous().to(DEV), uk.to(DEV), None, folded, heads, dim, rot, rank)
    assert torch.equal(folded[0], out[T - 1])


@pytest.mark.parametrize("heads, most", [(1, 1), (8, 2), (16, 1), (16, 4), (17, 1), (33, 1)])     # 1 to 64 rows an entry
@pytest.mark.parametrize("rot, page", [(0, 16), (16, 8), (64, 256), (64, 3)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("extras", [False, True])
def test_decoding_over_a_latent_of_512(heads, most, rot, page, window, extras):
    """Row tiles of 16 and 32, contexts at the edges of tiles of 64 keys, slices and none, pages given back behind a window, no
    number behind a context's last key; with sinks, score changes and a gate: against float64 over the rounded queries."""
    from safetyraise_lmengine_b200.kernels import ops
    rank, g = 512, torch.Generator().manual_seed(heads + rot + page)
    dk = rank + rot
    kv_lens = [64, 4, 65, 700, 129, 1]
    q_lens = [min(most, k) for k in kv_lens[:-1]] + [1]
    T, scale = sum(q_lens), 0.2
    ctx = Ctx(q_lens, kv_lens)
    from safetyraise_lmengine_b200.parts.base import Workspace
    ctx.n_entries, ctx.max_q_len, ctx.kv_bound, ctx.workspace = len(q_lens), max(q_lens), max(kv_lens), Workspace(torch.device(DEV), T)
    q = torch.randn(T, heads, dk, generator=g)
    keys = [torch.randn(k, dk, generator=g).bfloat16() for k in kv_lens]
    n_pages = sum(-(-k // page) for k in kv_lens)
    order, at = torch.randperm(n_pages, generator=g).tolist(), 0
    pool = torch.full((n_pages, 1, page, dk), float("nan"), dtype=torch.bfloat16)
    table = torch.full((len(kv_lens), max(-(-k // page) for k in kv_lens)), -1, dtype=torch.int32)
    for e, k in enumerate(kv_lens):
        first = max(0, k - q_lens[e] - window + 1) if window else 0
        for b in range(-(-k // page)):
            if (b + 1) * page <= first:
                continue                                                                # behind the window: given back
            table[e, b] = order[at]
            pool[order[at], 0, :min(page, k - b * page)] = keys[e][b * page:(b + 1) * page]
            at += 1
    sinks = torch.randn(heads, generator=g) if extras else None
    factor, weight, rate = torch.rand(heads, generator=g) + 0.5, torch.rand(heads, generator=g), torch.rand(heads, generator=g)
    logits = torch.randn(T, 3 + heads, generator=g)
    dev = lambda t: None if t is None else t.to(DEV)
    more = dict(head_scale=dev(factor), penalty=(dev(weight), dev(rate)), softcap=30.0, gate=(dev(logits), 3)) if extras else {}
    got = []
    for split in (True, False):
        out = torch.full((T, heads * rank), float("nan"), device=DEV)
        try:
            ops.split_general_attention = split
            ops.paged_attention_general(ctx, q.view(T, -1).to(DEV), pool.to(DEV), None, out, table.to(DEV), dev(sinks), heads, 1, dk, rank,
                                        scale, window, **more)
        finally:
            ops.split_general_attention = True
        got.append(out.cpu().double().view(T, heads, rank))
    assert ops.gemm_error_flag(out.device) == 0
    t = 0
    for e, (n, k) in enumerate(zip(q_lens, kv_lens)):
        x, c = q[t:t + n].bfloat16().double(), keys[e].double()
        i, j = torch.arange(k - n, k)[:, None], torch.arange(k)[None]
        s = torch.einsum("ihd,jd->hij", x, c) * scale
        if extras:
            s = 30.0 * torch.tanh(s * factor.double()[:, None, None] / 30.0)
            s = s - weight.double()[:, None, None] * torch.log1p(rate.double()[:, None, None] * (i - j).clamp(min=0))
        s = s.masked_fill((j > i) | ((window > 0) & (j <= i - window)), -math.inf)
        if extras:
            s = torch.cat([s, sinks.double()[:, None, None].expand(heads, n, 1)], -1)
        p = torch.softmax(s, -1)[..., :k]
        want, size = torch.einsum("hij,jd->ihd", p, c[:, :rank]), torch.einsum("hij,jd->ihd", p, c[:, :rank].abs())
        if extras:
            gate = torch.sigmoid(logits[t:t + n, 3:].double())[:, :, None]
            want, size = want * gate, size * gate
        for out in got:      # weights of 16 bits; scores of some 20 with float32 sums cut off a few dozen times
            assert ((out[t:t + n] - want).abs() <= 1e-4 * size + 1e-6).all(), e
        t += n

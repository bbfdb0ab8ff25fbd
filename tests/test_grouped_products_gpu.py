"""The grouped products of few rows an expert (mma.sync), the gather, the combination and the clamped GLU at the edges of
their tiles and vectors, against float64 loops."""
import pytest
import torch

from safetyraise_lmengine_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K", [8, 56, 64, 72, 264])          # around a slab of 64 and past the ring of four
@pytest.mark.parametrize("counts", [(1, 0, 16, 17), (32, 33, 48, 63), (64, 65, 0, 81)])
def test_rows_around_the_groups_of_sixteen(counts, K):
    g = torch.Generator().manual_seed(K + counts[0])
    E, N, n = len(counts), 136, sum(counts)
    choice = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])[torch.randperm(n, generator=g)]
    x = torch.randn(n, K, generator=g).bfloat16()
    w = torch.randn(E, N, K, generator=g).bfloat16()
    heads = torch.zeros(2, E + 1, dtype=torch.int32, device=DEV)
    por, rop = (torch.zeros(n, dtype=torch.int32, device=DEV) for _ in range(2))
    ops.moe_sort(choice[:, None].to(DEV), E, heads[0], heads[1], por, rop)
    out = torch.full((n, N), float("nan"), device=DEV)
    ops.moe_grouped(x.to(DEV), por, 1, w.to(DEV), out, heads[0], heads[1])
    got = out[rop.long()].cpu().double()
    for i in range(n):
        a, b = x[i].double(), w[int(choice[i])].double()
        # float32 sums of exact products: at most K roundings of the sum of the products' sizes
        assert ((got[i] - b @ a).abs() <= K * 2.0 ** -23 * (b.abs() @ a.abs())).all(), i


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,top", [(1, 4, 1), (3, 508, 4), (2, 512, 5), (5, 516, 9), (3, 515, 2)])
def test_combination_and_gather_and_activation(act, T, H, top):
    g = torch.Generator().manual_seed(H + top)
    n = T * top
    rows = torch.randn(n + 3, H, generator=g)
    rop = torch.randperm(n + 3, generator=g)[:n].to(torch.int32).reshape(T, top)
    rop[0, top - 1] = -1                                      # a pair without a row
    weight, shared = torch.rand(T, top, generator=g), torch.randn(T, H, generator=g).to(act)
    out = torch.empty(T, H, dtype=act, device=DEV)
    ops.moe_combine(rows.to(DEV), rop.to(DEV), weight.to(DEV), shared.to(DEV), out)
    w = torch.where(rop >= 0, weight, 0.).double()
    terms = w[..., None] * rows.double()[rop.clamp(min=0).long()]
    want, size = terms.sum(1) + shared.double(), terms.abs().sum(1) + shared.double().abs()
    step = 2.0 ** -24 if act == torch.float32 else 2.0 ** -8  # half the spacing of 24- and 8-bit significands over their least value
    assert ((out.cpu().double() - want).abs() <= (top + 2) * 2.0 ** -24 * size + step * want.abs()).all()
    got = torch.empty(T, H, device=DEV)
    both = torch.randn(T, 2 * H, generator=g)
    ops.clamped_glu(both.to(DEV), got, 1.2, 1.702)
    gate, up = both[:, :H].double().clamp(max=1.2), both[:, H:].double().clamp(-1.2, 1.2)
    assert torch.allclose(got.cpu().double(), gate * torch.sigmoid(1.702 * gate) * (up + 1), rtol=2e-6, atol=1e-9)
    if H % 4 == 0:
        x = torch.randn(T, 2 * H, generator=g).bfloat16()     # rows of a multiple of 8
        pair = torch.tensor([*range(n), -1], dtype=torch.int32)
        xs = torch.empty(n + 1, 2 * H, dtype=torch.bfloat16, device=DEV)
        ops.moe_gather_rows(x.to(DEV), pair.to(DEV), top, xs)
        assert torch.equal(xs.cpu(), torch.cat([x.repeat_interleave(top, 0), torch.zeros(1, 2 * H).bfloat16()]))


EPILOGUES = pytest.mark.parametrize("act, glu", [(None, False), ("gelu", False), ("relu_squared", False), (None, True)])
OUT_TYPES = pytest.mark.parametrize("odt", [torch.float32, torch.bfloat16])


@EPILOGUES
@OUT_TYPES
@pytest.mark.parametrize("tile, N, K, M", [(128, 256, 72, 800), (128, 512, 136, 768), (128, 768, 64, 1100), (256, 512, 72, 700),
                                           (256, 256, 64, 1), (128, 384, 72, 800), (128, 256, 72, 767), (128, 512, 64, 1)])
def test_tensor_memory_products_with_their_epilogues(act, glu, odt, tile, N, K, M):
    """Tiles of 256 tokens on pairs of SMs and of 128 on one (the weights fit the L2), with every epilogue: groups in any order,
    tiles without rows, a ragged last tile."""
    check_grouped(3, act, glu, odt, tile, N, K, M)


@EPILOGUES
@OUT_TYPES
@pytest.mark.parametrize("K, M", [(2056, 3109), (2048, 3072)])
def test_pairs_of_sms_on_tiles_of_128_tokens(act, glu, odt, K, M):
    """Weights of 64 Mi elements over all groups, and 192 rows a group (with its padding): tiles of 128 tokens on two SMs."""
    E, N = 16, 2048
    assert E * N * K >= 64 << 20 and M >= 192 * E
    check_grouped(E, act, glu, odt, 128, N, K, M)


def check_grouped(E, act, glu, odt, tile, N, K, M):
    tiles = -(-M // tile)
    g = torch.Generator(device=DEV).manual_seed(N + M)
    group = torch.tensor([[E - 1, -1, 0, 1][t % 4] if M > 1 else 1 for t in range(tiles)], dtype=torch.int32, device=DEV)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    out = torch.full((M, N // 2 if glu else N), 7.0, dtype=odt, device=DEV)
    ops.gemm_tn_tcgen05_grouped(x, w, out, group, glu=glu, limit=1.5, alpha=1.702, tile_rows=tile, act=act)
    assert ops.gemm_error_flag(out.device) == 0
    e = group.repeat_interleave(tile)[:M]
    rows = e >= 0
    assert (out[~rows] == 7.0).all()                          # tiles without a group are not written
    z, size = (torch.zeros(M, N, dtype=torch.float64, device=DEV) for _ in range(2))
    for k in e[rows].unique().tolist():
        z[e == k], size[e == k] = x[e == k].double() @ w[k].double().T, x[e == k].double().abs() @ w[k].double().abs().T
    err = K * 2.0 ** -23 * size                               # float32 sums of exact products
    if glu:
        z, err = z.view(M, N // 16, 2, 8), err.view(M, N // 16, 2, 8)
        gate, up = z[:, :, 0].clamp(max=1.5), z[:, :, 1].clamp(-1.5, 1.5)
        want = (gate * torch.sigmoid(1.702 * gate) * (up + 1)).reshape(M, -1)
        # gate * logistic(1.702 gate) below 1.5 has a slope below 1.11 and a size below 1.4; up + 1 lies below 2.5
        err = (2.8 * err[:, :, 0] + 1.4 * err[:, :, 1]).reshape(M, -1) + 2.0 ** -20
    elif act == "gelu":
        want, err = 0.5 * z * (1 + torch.erf(z / 2 ** 0.5)), 1.13 * err + z.abs() * 2.0 ** -21
    elif act == "relu_squared":
        want, err = z.clamp(min=0) ** 2, (2 * z.abs() + err) * err + z * z * 2.0 ** -23
    else:
        want = z
    err = err + (2.0 ** -24 if odt == torch.float32 else 2.0 ** -8) * want.abs()      # the result's own rounding
    assert ((out.double() - want).abs() <= err * 1.001)[rows].all()


@pytest.mark.parametrize("tile, N, K", [(128, 128, 64), (128, 512, 72), (256, 256, 136)])
@pytest.mark.parametrize("table", [[-1], [-1, -1, -1], [0] + [-1] * 40, [-1] * 33 + [1], [1, -1, 0] + [-1] * 70])
def test_tiles_behind_the_last_one_in_use(tile, N, K, table):
    """Tables with no group at all, with groups at their start or end, longer than a warp: the tiles of the groups are computed,
    the others' rows stay as they are."""
    g = torch.Generator().manual_seed(N + len(table))
    M = tile * len(table) - 5
    x, w = torch.randn(M, K, generator=g).bfloat16(), (torch.randn(2, N, K, generator=g) * K ** -0.5).bfloat16()
    out = torch.full((M, N), 7.0, device=DEV)
    ops.gemm_tn_tcgen05_grouped(x.to(DEV), w.to(DEV), out, torch.tensor(table, dtype=torch.int32, device=DEV), tile_rows=tile)
    assert ops.gemm_error_flag(out.device) == 0
    for t, group in enumerate(table):
        rows = slice(t * tile, min(M, (t + 1) * tile))
        got, a = out[rows].cpu(), x[rows].double()
        if group < 0:
            assert (got == 7.0).all()
        else:      # float32 sums of exact products, cut off or rounded K times
            assert ((got - a @ w[group].double().T).abs() <= K * 2.0 ** -23 * (a.abs() @ w[group].double().abs().T) + 1e-9).all()


# (the last three: more than 148 blocks with rows, whose rings are the short ones)
@pytest.mark.parametrize("T, E, top, F, K", [(*step, *size) for step in [(1, 3, 2), (16, 5, 3), (17, 4, 4), (32, 40, 2), (33, 2, 2), (64, 7, 3)]
                                             for size in [(8, 72), (72, 640), (128, 64), (136, 1032)]]
                         + [(16, 40, 3, 512, 328), (17, 40, 3, 512, 328), (33, 40, 2, 512, 328)])
@pytest.mark.parametrize("odt", [torch.float32, torch.bfloat16])
def test_experts_that_stream_their_weights(T, E, top, F, K, odt, monkeypatch):
    """Token tiles of 16, 32 and 64, experts without rows and with all tokens, features and k's that end inside a tile, rings of
    one block an SM and of three; rows by their tokens and packed, with every epilogue."""
    monkeypatch.setattr(type(ops), "experts_stream", staticmethod(lambda tokens, weight_elements: tokens > 0))
    g = torch.Generator().manual_seed(T + F)
    choice = torch.stack([torch.randperm(E - (E > 4), generator=g)[:top] for _ in range(T)])         # the last expert may have none
    flat = choice.flatten()
    order = torch.sort(flat, stable=True).indices.to(torch.int32)                                    # pair of row
    e = flat[order.long()]
    offsets = torch.tensor([int((e < k).sum()) for k in range(E + 1)], dtype=torch.int32)
    n, x = T * top, torch.randn(T, K, generator=g).bfloat16()
    packed = torch.randn(n, K, generator=g).bfloat16()
    scale = torch.rand(n, generator=g) + 0.5
    for glu, act, pairs, own in ((True, None, True, None), (True, None, True, scale), (False, None, False, None), (False, "gelu", True, None),
                                 (False, "relu_squared", False, None), (True, None, False, None)):
        w = (torch.randn(E, 2 * F if glu else F, K, generator=g) * K ** -0.5).bfloat16()
        out = torch.full((n, F), 7.0, dtype=odt, device=DEV)
        ops.moe_grouped((x if pairs else packed).to(DEV), order.to(DEV) if pairs else None, top if pairs else 1, w.to(DEV), out,
                        offsets.to(DEV), offsets.to(DEV), glu=glu, interleaved=glu, limit=1.5 if glu else 0.0, alpha=1.702 if glu else 0.0,
                        pair_scale=None if own is None else own.to(DEV), act=act, tokens=T)
        assert ops.gemm_error_flag(out.device) == 0
        rows = (x[order.long() // top] if pairs else packed).double()
        z = torch.einsum("rk,rnk->rn", rows, w[e].double())
        err = K * 2.0 ** -23 * torch.einsum("rk,rnk->rn", rows.abs(), w[e].double().abs())           # float32 sums of exact products
        if own is not None:
            z, err = z * own[order.long()].double()[:, None], err * own[order.long()].double()[:, None] + z.abs() * 2.0 ** -22
        if glu:
            z, err = z.view(n, F // 8, 2, 8), err.view(n, F // 8, 2, 8)
            gate, up = z[:, :, 0].clamp(max=1.5), z[:, :, 1].clamp(-1.5, 1.5)
            want = (gate * torch.sigmoid(1.702 * gate) * (up + 1)).reshape(n, -1)
            err = (2.8 * err[:, :, 0] + 1.4 * err[:, :, 1]).reshape(n, -1) + 2.0 ** -20              # slopes and sizes as above
        elif act == "gelu":
            want, err = 0.5 * z * (1 + torch.erf(z / 2 ** 0.5)), 1.13 * err + z.abs() * 2.0 ** -21
        elif act == "relu_squared":
            want, err = z.clamp(min=0) ** 2, (2 * z.abs() + err) * err + z * z * 2.0 ** -23
        else:
            want = z
        err = err + (2.0 ** -24 if odt == torch.float32 else 2.0 ** -8) * want.abs()
        assert ((out.cpu().double() - want).abs() <= err * 1.001).all(), (glu, act, pairs)

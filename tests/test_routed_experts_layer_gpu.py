"""Layers of routed experts as a decoder builds them, at the lines between the forms of their products and with choices that are
no ordinary ones, against float64 loops."""
import math

import pytest
import torch

from safetyraise_lmengine_b200.config.spec import RoutedExpertsSpec
from safetyraise_lmengine_b200.kernels import ops
from safetyraise_lmengine_b200.parts import FEED_FORWARDS, ModelContext, StepContext, Workspace

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Layer:
    """A layer in bfloat16, its weights, and what it computes in float64 for a given choice."""

    def __init__(self, seed, experts, top, hidden, inner, vocab=0, table=None, bias=None, **more):
        g = torch.Generator().manual_seed(seed)
        mat = lambda *s: (torch.randn(*s, generator=g) * 1.5 * s[-1] ** -0.5).bfloat16()
        self.spec = RoutedExpertsSpec(kind="routed_experts", hidden_size=hidden, intermediate_size=inner, activation="silu",
                                      experts=experts, top=top, router_bias=bias is not None, vocab=vocab, **more)
        w = {"mlp.router": mat(experts, hidden)} if table is None else {"mlp.table": table}
        if bias is not None:
            w["mlp.router.b"] = bias
        for e in range(experts):
            w.update({f"mlp.e{e}.gate": mat(inner, hidden), f"mlp.e{e}.up": mat(inner, hidden), f"mlp.e{e}.down": mat(hidden, inner)})
        self.w = w
        self.part = FEED_FORWARDS["routed_experts"](self.spec, "", {n: t.to(DEV) for n, t in w.items()},
                                                    ModelContext(torch.device(DEV), torch.bfloat16, 4096, {}))

    def run(self, x, ids=None):
        T = x.shape[0]
        ctx = StepContext(T=T, n_entries=T, token_ids=None if ids is None else ids.to(DEV), positions=None, entry_of_token=None, slots=None,
                          cu_q=None, kv_lens=None, logit_rows=None, block_tables={}, kv_slot={}, host={}, cache=None,
                          workspace=Workspace(torch.device(DEV), T), dtype=torch.bfloat16)
        out = self.part.forward(ctx, x.to(DEV)).cpu().double()
        assert ops.gemm_error_flag(torch.device(DEV)) == 0
        return out

    def exact(self, x, choice, weight):
        """-> (the layer's output, how far a bfloat16 layer with float32 sums may be from it), for choice and weight [T, top]."""
        on_input = self.spec.weight_on_input
        out, err = torch.zeros(x.shape, dtype=torch.float64), torch.zeros(x.shape, dtype=torch.float64)
        for e in range(self.spec.experts):
            gate, up, down = (self.w[f"mlp.e{e}.{n}"].double() for n in ("gate", "up", "down"))
            for c in range(choice.shape[1]):
                t = (choice[:, c] == e).nonzero()[:, 0]
                own = weight[t, c, None]
                a = x[t].double() * (own if on_input else 1)
                z, u = a @ gate.T, a @ up.T
                zs, us = a.abs() @ gate.abs().T, a.abs() @ up.abs().T
                y = z * torch.sigmoid(z) * u
                # float32 sums cut off or rounded once a product; slope of the silu at most 1.1; y is rounded to 8 bits
                y_err = a.shape[1] * 2.0 ** -23 * (1.1 * zs * u.abs() + us * z.abs()) + 2.0 ** -21 * y.abs()
                y_err = y_err + 2.0 ** -9 * (y.abs() + y_err)
                scale = 1 if on_input else own
                out[t] += scale * (y @ down.T)
                err[t] += scale * ((y_err + y.shape[1] * 2.0 ** -23 * y.abs()) @ down.abs().T)
        return out, (err + 2.0 ** -9 * (out.abs() + err)) * 1.001 + 1e-9


@pytest.mark.parametrize("scoring", ["softmax_of_chosen", "logistic", "softmax_over_all"])
def test_a_router_names_no_expert_twice(scoring):
    inf, nan = math.inf, math.nan
    rows = [[1.0, 3.0, 2.0, 0.0, -1.0, 0.5], [-inf, -inf, 4.0, -inf, -inf, -inf], [-inf] * 6, [nan] * 6, [nan, 2.0, nan, nan, 1.0, nan],
            [5.0, nan, -inf, nan, nan, nan], [-inf, nan, 0.0, nan, -inf, 1.0]]
    want = [[1, 2, 0, 5], [2, 0, 1, 3], [0, 1, 2, 3], [0, 1, 2, 3], [1, 4, 0, 2], [0, 2, 1, 3], [5, 2, 0, 4]]
    z = torch.tensor(rows, device=DEV)
    T, E, top = z.shape[0], z.shape[1], 4
    i32 = lambda *s: torch.zeros(*s, dtype=torch.int32, device=DEV)
    for route in (True, False):
        choice, weight = i32(T, top), torch.zeros(T, top, device=DEV)
        if route:
            ops.moe_route(z, None, top, choice, weight, scoring=scoring)
        else:
            ops.moe_sort(choice, E, i32(E + 1), i32(E + 1), i32(T * top), i32(T * top), route=(z, 0, None, weight), scoring=scoring)
        assert choice.tolist() == want
        assert (weight[1, 1:] == 0).all() and weight[0].isfinite().all()


def test_experts_whose_choice_is_masked_out_or_named_twice():
    """A bias of -inf leaves fewer experts than a token takes; a table (not one that the loader would take) names an expert twice:
    every row of the experts' products is formed all the same."""
    g = torch.Generator().manual_seed(3)
    E, top, H, I, T = 5, 3, 72, 40, 9
    x = torch.randn(T, H, generator=g).bfloat16()
    bias = torch.tensor([-math.inf, 0.5, -math.inf, -math.inf, -math.inf])
    layer = Layer(1, E, top, H, I, bias=bias)
    want, err = layer.exact(x, torch.full((T, 1), 1), torch.ones(T, 1, dtype=torch.float64))
    assert ((layer.run(x) - want).abs() <= err).all()
    table = torch.tensor([[4, 4, 1], [0, 2, 0], [3, 3, 3], [1, 2, 3]], dtype=torch.int32)
    layer = Layer(2, E, top, H, I, vocab=4, table=table, scoring="table")
    ids = torch.tensor([0, 1, 2, 2, 2, 2, 2, 3, 0], dtype=torch.int32)
    want, err = layer.exact(x, table[ids.long()], torch.full((T, top), 1 / top, dtype=torch.float64))
    assert ((layer.run(x, ids) - want).abs() <= err).all()


@pytest.mark.parametrize("T", [60, 90, 100, 127, 128, 200])
def test_a_weight_on_the_input_costs_no_bits_below_whole_tiles(T):
    """Below 64 rows an expert the weight multiplies float32 sums, so that only the products' inner result and the output are
    rounded to 8 bits (each by 2^-9 of an element at most, independently of each other); from there on the input is, too."""
    g = torch.Generator().manual_seed(T)
    E, H, I = 2, 256, 256
    layer = Layer(5, E, 1, H, I, scoring="logistic", weight_on_input=True)
    x = torch.randn(T, H, generator=g).bfloat16()
    z = x.double() @ layer.w["mlp.router"].double().T
    weight, choice = torch.sigmoid(z).max(1, keepdim=True)
    want, _ = layer.exact(x, choice, weight)
    off = float((layer.run(x) - want).norm() / want.norm())
    print("rows an expert", T / E, "error", off)
    assert off <= 2 ** -9 * (2 ** 0.5 if T < 64 * E else 3)


# 16 and 64 tokens: the experts' weights are streamed past all tokens up to there (64: from 2 Mi elements a matrix on, here the first
# product alone); 36 and 44 rows an expert: whole tiles from there on
@pytest.mark.parametrize("H, I, lines", [(256, 256, (16, 88)), (1024, 1024, (16, 64, 88)), (1024, 2048, (16, 64, 72))])
def test_a_token_on_either_side_of_the_lines_between_the_forms(H, I, lines):
    """The forms of the experts' products round at the same places: below and above each line a token's output is within the
    roundings' bound of float64."""
    E, top = 4, 2
    layer = Layer(7, E, top, H, I)
    x = torch.randn(max(lines) + 1, H, generator=torch.Generator().manual_seed(H + I)).bfloat16()
    value, choice = (x.double() @ layer.w["mlp.router"].double().T).topk(top, 1)
    want, err = layer.exact(x, choice, torch.softmax(value, 1))
    assert [ops.experts_stream(t, 2 * I * H) for t in (16, 17, 64, 65)] == [True, I * H >= 1 << 20, I * H >= 1 << 20, False]
    assert [ops.grouped_takes_tiles(top * t, E, 2 * I * H) for t in (max(lines) - 1, max(lines))] == [False, True]
    for T in sorted({t + d for t in lines for d in (-1, 0, 1)}):
        assert ((layer.run(x[:T]) - want[:T]).abs() <= err[:T]).all(), T

"""The work that the engine is timed on: what a program that serves models with it has it do, layer by layer and in whole
steps.

Layers are built from their specifications the way the decoder builds them (the registries of ``parts``) and run on a
step's context with a paged cache behind it.  Decode steps replay a CUDA graph recorded once, as the engine's step
function does; prompts and mixed steps are launched kernel by kernel, as it does too.  Two cases are whole steps
through ``Engine.step`` and return logits.

Sizes: the Qwen3 layer sizes of the benchmark configurations (8B, 14B, 32B), the layers of 1,024 to 4,096 wide that
``bench.py --design`` times for the other architectures, pages of 16 tokens, contexts up to 4,096 tokens.
"""
import math
import random

import torch

from safetyraise_lmengine_b200 import Engine, SamplingParams, StepEntry
from safetyraise_lmengine_b200.cache.manager import FIXED_STATE, CacheGroupSpec, CacheManager
from safetyraise_lmengine_b200.config.spec import (AttentionSpec, DeltaRuleSpec, FeedForwardSpec, LatentAttentionSpec,
                                                   LayerSpec, NormSpec, PositionSpec, RoutedExpertsSpec, RunStep,
                                                   SelectiveScanSpec)
from safetyraise_lmengine_b200.kernels import ops
from safetyraise_lmengine_b200.parts import (BLOCKS, FEED_FORWARDS, MIXERS, NORMS, ModelContext, StepContext,
                                             Workspace)
from safetyraise_lmengine_b200.sampling.sampler import Sampler

PAGE = 16
HEAD = 128                   # head size of every attention here
KV_HEADS = 8                 # of the Qwen3 layers
EPS = 1e-6
ROWS = 4096                  # rows of the embedding table in front of a layer
VOCAB = 32768                # of a whole step in bfloat16
DEV = "cuda"

SHAPES = {"8b": (4096, 32, 12288), "14b": (5120, 40, 17408), "32b": (5120, 64, 25600)}   # hidden, heads, feed-forward


def listed():
    return [
        # a Qwen3-8B layer while one user is answered: the smallest piece of work, all latency and weights
        {"name": "layer_decode_1", "kind": "layer_decode", "shape": "8b", "batch": 1, "context": 2048},
        # a whole decode step of a full batch, layers of 8B sizes, logits of every request
        {"name": "step_decode_64", "kind": "step_decode", "layers": 4, "batch": 64, "context": 2048},
        # a prompt of 2,048 tokens through a layer of 8B sizes: the headline prefill
        {"name": "layer_prompt_2048", "kind": "layer_prompt", "shape": "8b", "tokens": 2048, "start": 0, "decodes": 0,
         "context": 0},
        # a portion of a prompt beside decoding requests, 14B sizes: the mixed steps of chunked prefill
        {"name": "layer_portion_481_beside_31", "kind": "layer_prompt", "shape": "14b", "tokens": 481, "start": 512,
         "decodes": 31, "context": 1500},
        # attention over a cached latent: a prompt behind a short shared beginning, and a decode batch
        {"name": "latent_prompt_1800", "kind": "latent_prompt", "width": 2048, "tokens": 1800, "start": 200},
        {"name": "latent_decode_8", "kind": "latent_decode", "width": 2048, "batch": 8, "context": 2048},
        # the gated delta rule on three prompts of unlike lengths
        {"name": "delta_prompts_2000", "kind": "delta_prompt", "width": 2048, "tokens": 2000, "requests": 3},
        # the selective scan on one long prompt
        {"name": "scan_prompt_2048", "kind": "scan_prompt", "width": 2048, "tokens": 2048, "requests": 1},
        # routed experts beside a shared one: a prompt, and a decode batch
        {"name": "experts_prompt_2048", "kind": "experts", "width": 2048, "tokens": 2048},
        {"name": "experts_decode_8", "kind": "experts", "width": 2048, "tokens": 8},
        # temperature, top-k, top-p and a repetition penalty over the full vocabulary, tokens back on the host
        {"name": "sampling_8", "kind": "sampling", "batch": 8, "vocab": 151936, "top_k": 50, "top_p": 0.9,
         "penalty": 1.1},
        # the true 32-bit path: a whole step of a small Qwen3, a portion of a prompt beside decoding requests
        {"name": "step_float32_300_beside_5", "kind": "step_float32", "layers": 3, "hidden": 1024, "heads": 16,
         "kv_heads": 8, "head_dim": 64, "inter": 3072, "vocab": 8192, "tokens": 300, "decodes": 5, "context": 700},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["layer_decode", "step_decode", "layer_prompt", "latent_prompt", "latent_decode", "delta_prompt",
                       "scan_prompt", "experts", "sampling", "step_float32"])
    width = rng.choice([1024, 2048, 4096])
    if kind == "layer_decode":
        return {"kind": kind, "shape": rng.choice(list(SHAPES)), "batch": _spread(rng, 1, 64), "context": _spread(rng, 16, 4000)}
    if kind == "step_decode":
        return {"kind": kind, "layers": rng.randint(2, 4), "batch": _spread(rng, 1, 64), "context": _spread(rng, 16, 2048)}
    if kind == "layer_prompt":
        shape = rng.choice(["8b", "14b"])
        tokens = _spread(rng, 5, 2048 if shape == "8b" else 1024)
        decodes = rng.choice([0, 0, rng.randint(1, 32)])
        return {"kind": kind, "shape": shape, "tokens": tokens, "start": rng.choice([0, rng.randint(1, 2000)]),
                "decodes": decodes, "context": _spread(rng, 16, 2048) if decodes else 0}
    if kind == "latent_prompt":
        return {"kind": kind, "width": width, "tokens": _spread(rng, 5, 2048), "start": rng.choice([0, rng.randint(1, 1000)])}
    if kind == "latent_decode":
        return {"kind": kind, "width": width, "batch": _spread(rng, 1, 64), "context": _spread(rng, 16, 4000)}
    if kind in ("delta_prompt", "scan_prompt"):
        requests = rng.randint(1, 4)
        return {"kind": kind, "width": width, "tokens": max(5 * requests, _spread(rng, 5, 2048)), "requests": requests}
    if kind == "experts":
        return {"kind": kind, "width": width, "tokens": _spread(rng, 1, 2048)}
    if kind == "sampling":
        return {"kind": kind, "batch": _spread(rng, 1, 64), "vocab": _spread(rng, 32000, 151936),
                "top_k": rng.choice([0, 1, rng.randint(2, 200)]), "top_p": round(rng.uniform(0.5, 1.0), 3),
                "penalty": rng.choice([1.0, 1.1])}
    head_dim = rng.choice([64, 128])
    kv = rng.choice([2, 4])
    return {"kind": kind, "layers": rng.randint(1, 3), "hidden": rng.choice([512, 768, 1000]), "heads": 2 * kv, "kv_heads": kv,
            "head_dim": head_dim, "inter": rng.choice([1536, 2500]), "vocab": 2 * _spread(rng, 1000, 4000),
            "tokens": _spread(rng, 1, 400), "decodes": rng.randint(1, 8), "context": _spread(rng, 16, 1000)}


# ---- sizes that follow from a case ------------------------------------------------------------------------------

def _ragged(count, most, salt):
    """``count`` context lengths between half of ``most`` and ``most``, the longest among them; the same for every seed."""
    rng = random.Random(f"{count}:{most}:{salt}")
    return [most] + [rng.randint(max(1, most // 2), most) for _ in range(count - 1)] if count else []


def _shares(total, parts, salt):
    """``total`` tokens in ``parts`` prompts of unlike lengths."""
    rng = random.Random(f"{total}:{parts}:{salt}")
    cuts = sorted(rng.sample(range(1, total), parts - 1)) if parts > 1 else []
    return [b - a for a, b in zip([0] + cuts, cuts + [total])]


def _batch(case):
    """(new tokens, tokens already held) of every request of the case's step."""
    k = case["kind"]
    if k in ("layer_decode", "step_decode", "latent_decode"):
        return [(1, n) for n in _ragged(case["batch"], case["context"], k)]
    if k == "layer_prompt":
        return [(1, n) for n in _ragged(case["decodes"], case["context"], k)] + [(case["tokens"], case["start"])]
    if k == "step_float32":
        return [(1, n) for n in _ragged(case["decodes"], case["context"], k)] + [(case["tokens"], 0)]
    if k == "latent_prompt":
        return [(case["tokens"], case["start"])]
    return [(n, 0) for n in _shares(case["tokens"], case["requests"], k)]


def _pairs(batch):
    """Pairs of a query and a key that it sees."""
    return sum(q * s + q * (q + 1) // 2 for q, s in batch)


def _qwen(case):
    """(layers, hidden, heads, KV heads, head size, feed-forward) of a Qwen3 case."""
    if case["kind"] == "step_float32":
        return tuple(case[k] for k in ("layers", "hidden", "heads", "kv_heads", "head_dim", "inter"))
    h, n, i = SHAPES[case.get("shape", "8b")]
    return case.get("layers", 1), h, n, KV_HEADS, HEAD, i


def _latent(case):
    """(heads, head size, rotated size, value size, rank): heads of 128 + 64, a latent of 512."""
    return case["width"] // HEAD, HEAD, 64, HEAD, 512


def _scan(case):
    """(channels, states, rank of the step sizes, taps)."""
    return 2 * case["width"], 16, case["width"] // 16, 4


EXPERTS, TOP, LIMIT, ALPHA, TAPS = 16, 4, 7.0, 1.702, 4


# ---- weights and inputs, from the seed alone --------------------------------------------------------------------

class _Draws:
    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(1000003 * seed + 17)

    def normal(self, shape, scale=1.0, dtype=torch.bfloat16):
        out = torch.empty(shape, dtype=dtype, device=DEV)
        flat = out.view(-1)
        for lo in range(0, flat.numel(), 1 << 26):
            part = flat[lo:lo + (1 << 26)]
            part.copy_(torch.randn(part.numel(), generator=self.gen, device=DEV) * scale)
        return out

    def matrix(self, *shape):
        return self.normal(shape, 0.02)

    def scale(self, n):
        return 1.0 + 0.1 * torch.randn(n, generator=self.gen, device=DEV)

    def uniform(self, n, lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=self.gen, device=DEV)

    def ids(self, n, below):
        return torch.randint(0, below, (n,), generator=self.gen, device=DEV, dtype=torch.int32)


def _step_bias(d, n):
    """Biases ahead of a softplus that give step sizes between 0.001 and 0.1, spread over their logarithm."""
    dt = torch.exp(d.uniform(n, math.log(1e-3), math.log(1e-1)))
    return dt + torch.log(-torch.expm1(-dt))


def _qwen_layer_weights(d, p, hidden, heads, kv, hd, inter):
    w = {p + "input_layernorm.weight": d.scale(hidden), p + "post_attention_layernorm.weight": d.scale(hidden),
         p + "self_attn.q_norm.weight": d.scale(hd), p + "self_attn.k_norm.weight": d.scale(hd),
         p + "self_attn.q_proj.weight": d.matrix(heads * hd, hidden), p + "self_attn.k_proj.weight": d.matrix(kv * hd, hidden),
         p + "self_attn.v_proj.weight": d.matrix(kv * hd, hidden), p + "self_attn.o_proj.weight": d.matrix(hidden, heads * hd),
         p + "mlp.gate_proj.weight": d.matrix(inter, hidden), p + "mlp.up_proj.weight": d.matrix(inter, hidden),
         p + "mlp.down_proj.weight": d.matrix(hidden, inter)}
    return w


def _inputs(case, seed):
    """Everything random of a case: weights by name, token ids or the layer's input, what the cache holds already."""
    k, d = case["kind"], _Draws(seed)
    if k == "sampling":
        B, V = case["batch"], case["vocab"]
        hist = torch.randint(0, V, (B, 100), generator=d.gen, device=DEV).tolist()
        return {"logits": d.normal((B, V), 3.0, torch.float32), "seeds": [int(t) for t in d.ids(B, 1 << 30)], "history": hist}
    if k in ("layer_decode", "layer_prompt", "step_decode", "step_float32"):
        layers, hidden, heads, kv, hd, inter = _qwen(case)
        whole = k.startswith("step")
        batch = _batch(case)
        w = {}
        for i in range(layers):
            w.update(_qwen_layer_weights(d, f"model.layers.{i}.", hidden, heads, kv, hd, inter))
        rows = (case["vocab"] if k == "step_float32" else VOCAB) if whole else ROWS
        # in front of one layer the stream has the size that a stack's middle has
        w["model.embed_tokens.weight"] = d.normal((rows, hidden), 0.02 if whole else 1.0)
        w["model.norm.weight"] = d.scale(hidden)
        if whole:
            w["lm_head.weight"] = d.matrix(rows, hidden)
        dtype = torch.float32 if k == "step_float32" else torch.bfloat16
        held = sum(s for _, s in batch)
        return {"w": w, "ids": d.ids(sum(q for q, _ in batch), rows),
                "cache": [[d.normal((held, kv, hd), 1.0, dtype) for _ in range(2)] for _ in range(layers)]}
    W = case["width"]
    if k == "experts":
        I = W // 2
        w = {"mlp.router": d.matrix(EXPERTS, W), "mlp.router.b": d.normal((EXPERTS,), 0.1, torch.float32)}
        for e in ["e%d." % e for e in range(EXPERTS)] + ["shared."]:
            n = W if e == "shared." else I
            w.update({"mlp." + e + "gate": d.matrix(n, W), "mlp." + e + "up": d.matrix(n, W), "mlp." + e + "down": d.matrix(W, n)})
        return {"w": w, "x": d.normal((case["tokens"], W))}
    batch = _batch(case)
    x = d.normal((sum(q for q, _ in batch), W))
    if k.startswith("latent"):
        H, dim, rot, dv, rank = _latent(case)
        w = {"mix.q": d.matrix(H * (dim + rot), W), "mix.dkv": d.matrix(rank + rot, W), "mix.dkv.norm": d.scale(rank),
             "mix.uk": d.matrix(H * dim, rank), "mix.uv": d.matrix(H * dv, rank), "mix.g": d.matrix(H, W), "mix.o": d.matrix(W, H * dv)}
        return {"w": w, "x": x, "cache": d.normal((sum(s for _, s in batch), rank + rot))}
    if k == "delta_prompt":
        H = W // HEAD
        w = {}
        for n in "qkv":
            w["mix." + n] = d.matrix(H * HEAD, W)
            w["mix." + n + ".conv"] = d.normal((H * HEAD, TAPS), 0.4)
        w.update({"mix.b": d.matrix(H, W), "mix.a": d.matrix(H, W), "mix.A_log": torch.log(d.uniform(H, 1.0, 16.0)),
                  "mix.dt_bias": _step_bias(d, H), "mix.norm": d.scale(HEAD), "mix.g": d.matrix(H * HEAD, W),
                  "mix.o": d.matrix(W, H * HEAD)})
        return {"w": w, "x": x}
    C, N, R, taps = _scan(case)
    w = {"mix.in": d.matrix(2 * C, W), "mix.conv": d.normal((C, taps), 0.4, torch.float32),
         "mix.conv.b": d.normal((C,), 0.1, torch.float32), "mix.x": d.matrix(R + 2 * N, C), "mix.dt": d.normal((C, R), R ** -0.5),
         "mix.dt.b": _step_bias(d, C), "mix.A_log": torch.log(torch.arange(1, N + 1, device=DEV).float()).expand(C, N).contiguous(),
         "mix.D": d.scale(C), "mix.o": d.matrix(W, C)}
    return {"w": w, "x": x}


# ---- the framework's side: a part, its cache, a step's context ---------------------------------------------------

def _rotary(dims, base, kind="rotary_half"):
    return PositionSpec(kind, base, dims, dims)


def _mixer_spec(case):
    k, W = case["kind"], case.get("width")
    if k.startswith("latent"):
        H, dim, rot, dv, rank = _latent(case)
        return LatentAttentionSpec(kind="latent_attention", hidden_size=W, heads=H, head_dim=dim, rot_dim=rot, v_head_dim=dv,
                                   kv_rank=rank, softmax_scale=(dim + rot) ** -0.5, latent_norm_eps=EPS,
                                   position=_rotary(rot, 10000.0, "rotary_interleaved"))
    if k == "delta_prompt":
        return DeltaRuleSpec(kind="delta_rule", hidden_size=W, heads=W // HEAD, kv_heads=W // HEAD, head_dim=HEAD,
                             v_head_dim=HEAD, conv_taps=TAPS, norm_eps=EPS, unit_eps=EPS)
    C, N, R, taps = _scan(case)
    return SelectiveScanSpec(kind="selective_scan", hidden_size=W, inner=C, state=N, dt_rank=R, conv_taps=taps)


def _layer_spec(case):
    _, hidden, heads, kv, hd, inter = _qwen(case)
    mixer = AttentionSpec(kind="paged_attention", hidden_size=hidden, heads=heads, kv_heads=kv, head_dim=hd,
                          qk_norm=NormSpec("rmsnorm", hd, EPS), position=_rotary(hd, 1e6), softmax_scale=hd ** -0.5)
    norm = NormSpec("rmsnorm", hidden, EPS)
    return LayerSpec("pre_norm", mixer, FeedForwardSpec("gated_dense", hidden, inter), norm, norm, "model.layers.0.")


def _cache_for(need, batch):
    pages = sum(-(-(q + s) // PAGE) for q, s in batch) + 1
    group = CacheGroupSpec(name="g", kind=need.kind, entries=(0,), kv_heads=need.kv_heads, head_dim=need.head_dim,
                           window=need.window, state_shape=need.state_shape, state_dtype=need.state_dtype,
                           v_head_dim=need.v_head_dim)
    return CacheManager([group], PAGE, pages, len(batch), torch.bfloat16, torch.device(DEV))


def _context(cache, batch, ids=None):
    """A step's context over the requests of ``batch``, and the flat cache rows of the tokens that they hold already."""
    paged = bool(cache.paged_groups)
    slots = [cache.open_request() for _ in batch]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    T = sum(q for q, _ in batch)
    lens = [q + s for q, s in batch]
    tables, kv_slot, held = {}, {}, []
    if paged:
        width = -(-(-(-max(lens) // PAGE)) // 16) * 16          # decode steps round their tables' width like the engine
        table = torch.zeros(len(batch), width, dtype=torch.int32)
        rows = []
        for e, (slot, (q, s)) in enumerate(zip(slots, batch)):
            assert cache.reserve(slot, q + s)
            if s:
                cache.commit(slot, s)
            mine = cache.table("g", slot)
            table[e, :len(mine)] = torch.tensor(mine, dtype=torch.int32)
            row = [mine[p // PAGE] * PAGE + p % PAGE for p in range(q + s)]
            held += row[:s]
            rows += row[s:]
        tables, kv_slot = {"g": table.to(DEV)}, {"g": i32(rows)}
    bound = width * PAGE if paged else max(lens)
    cu = [0]
    for q, _ in batch:
        cu.append(cu[-1] + q)
    ctx = StepContext(
        T=T, n_entries=len(batch), token_ids=ids if ids is not None else i32([0] * T),
        positions=i32([s + j for q, s in batch for j in range(q)]),
        entry_of_token=i32([e for e, (q, _) in enumerate(batch) for _ in range(q)]), slots=i32(slots), cu_q=i32(cu),
        kv_lens=i32(lens), logit_rows=i32([c - 1 for c in cu[1:]]), block_tables=tables, kv_slot=kv_slot,
        host={"q_lens": [q for q, _ in batch], "starts": [s for _, s in batch], "kv_lens": lens, "slots": slots},
        cache=cache, workspace=Workspace(torch.device(DEV), T), dtype=torch.bfloat16, max_q_len=max(q for q, _ in batch),
        max_kv_len=max(lens), kv_bound=bound)
    return ctx, held


def _put(pool, rows, values):
    """Writes [tokens, heads, size] into a pool of pages [pages, heads, page, size] at flat rows page * PAGE + place."""
    if rows:
        at = torch.tensor(rows, device=DEV)
        pool[at // PAGE, :, at % PAGE] = values.to(pool.dtype)


class _Source:
    """A model's tensors, by name."""
    def __init__(self, tensors):
        self.tensors = tensors

    def names(self):
        return self.tensors.keys()

    def meta(self, name):
        t = self.tensors[name]
        return t.dtype, tuple(t.shape), t.numel() * t.element_size()

    def get(self, name):
        return self.tensors[name]


def _prepare_step(case, inp):
    layers, hidden, heads, kv, hd, inter = _qwen(case)
    f32 = case["kind"] == "step_float32"
    batch = _batch(case)
    T = sum(q for q, _ in batch)
    config = {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": layers, "hidden_size": hidden,
              "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": hd, "intermediate_size": inter,
              "vocab_size": inp["w"]["lm_head.weight"].shape[0], "rope_theta": 1e6, "rms_norm_eps": EPS,
              "tie_word_embeddings": False, "max_position_embeddings": 4096}
    pages = sum(-(-(q + s) // PAGE) for q, s in batch) + 1
    eng = Engine.from_source(config, _Source(inp["w"]), dtype="float32" if f32 else "bfloat16", device=DEV + ":0", page_size=PAGE,
                             num_pages=pages, max_requests=len(batch), max_batch_tokens=T, max_context=4096)
    slots, rows = [], []
    for q, s in batch:
        slot = eng.open_request()
        if s:
            assert eng.cache.reserve(slot, s)
            eng.cache.commit(slot, s)
            table = eng.cache.table(eng.cache.paged_groups[0].name, slot)
            rows += [table[p // PAGE] * PAGE + p % PAGE for p in range(s)]
        slots.append(slot)
    for i, (k, v) in enumerate(inp["cache"]):
        for pool, values in zip(eng.cache.kv_of_entry(i)[:2], (k, v)):
            _put(pool, rows, values)
    ids, entries, at = inp["ids"].tolist(), [], 0
    for slot, (q, s) in zip(slots, batch):
        entries.append(StepEntry(slot, ids[at:at + q], [q - 1]))
        at += q
    return {"kind": case["kind"], "engine": eng, "entries": entries, "starts": [s for _, s in batch]}


def _recorded(state, once):
    """A state whose pass is the replay of a CUDA graph of ``once``."""
    for _ in range(2):
        once(state)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        state["out"] = once(state)
    state["graph"] = graph
    return state


def prepare(case, seed):
    inp = _inputs(case, seed)
    k = case["kind"]
    if k == "sampling":
        params = SamplingParams(temperature=0.8, top_k=case["top_k"], top_p=case["top_p"], repetition_penalty=case["penalty"])
        return {"kind": k, "sampler": Sampler(torch.device(DEV), case["vocab"], max_rows=case["batch"]), **inp,
                "params": [params] * case["batch"], "indices": [3] * case["batch"]}
    if k.startswith("step"):
        return _prepare_step(case, inp)
    batch = _batch(case) if k != "experts" else [(1, 0)] * case["tokens"]
    T = sum(q for q, _ in batch)
    mctx = ModelContext(torch.device(DEV), torch.bfloat16, T, {})
    if k == "experts":
        W = case["width"]
        spec = RoutedExpertsSpec(kind="routed_experts", hidden_size=W, intermediate_size=W // 2, activation="clamped_glu",
                                 experts=EXPERTS, top=TOP, limit=LIMIT, glu_alpha=ALPHA, shared_size=W, shared_limit=LIMIT)
        state = {"kind": k, "part": FEED_FORWARDS[spec.kind](spec, "", inp["w"], mctx), "x": inp["x"],
                 "ctx": StepContext(T=T, n_entries=T, token_ids=None, positions=None, entry_of_token=None, slots=None, cu_q=None,
                                    kv_lens=None, logit_rows=None, block_tables={}, kv_slot={}, host={}, cache=None,
                                    workspace=Workspace(torch.device(DEV), T), dtype=torch.bfloat16)}
        return _recorded(state, _experts_pass) if T <= 64 else state
    if k in ("layer_decode", "layer_prompt"):
        spec = _layer_spec(case)
        block = BLOCKS[spec.block](spec, inp["w"], mctx)
        cache = _cache_for(block.mixer.cache_need(), batch)
        ctx, held = _context(cache, batch, inp["ids"])
        for pool, values in zip(cache.kv_of_entry(0)[:2], inp["cache"][0]):
            _put(pool, held, values)
        norm = NormSpec("rmsnorm", spec.mixer_norm.size, EPS)
        state = {"kind": k, "block": block, "norm": NORMS[norm.kind](norm, "model.norm.weight", inp["w"], mctx), "ctx": ctx,
                 "table": inp["w"]["model.embed_tokens.weight"], "flag": torch.zeros(1, dtype=torch.int32, device=DEV),
                 "residual": torch.empty(T, norm.size, device=DEV),
                 "normed": torch.empty(T, norm.size, dtype=torch.bfloat16, device=DEV)}
        return _recorded(state, _layer_pass) if k == "layer_decode" else state
    spec = _mixer_spec(case)
    part = MIXERS[spec.kind](spec, "", inp["w"], mctx)
    cache = _cache_for(part.cache_need(), batch)
    ctx, held = _context(cache, batch)
    state = {"kind": k, "part": part, "ctx": ctx, "x": inp["x"]}
    if "cache" in inp:
        _put(cache.kv_of_entry(0)[0], held, inp["cache"][:, None])
        state["pages"] = cache.kv_of_entry(0)[0]
    else:
        assert part.cache_need().kind == FIXED_STATE
        state["state"] = cache.state_of_entry(0)
    return _recorded(state, _latent_pass) if k == "latent_decode" else state


# ---- one pass ------------------------------------------------------------------------------------------------------

RUN = RunStep(0, 0, True)


def _layer_pass(s):
    """The token rows, a block, and the norm behind it (of the next block, or the final one)."""
    ops.embed_gather(s["ctx"].token_ids, s["table"], s["residual"], s["flag"])
    pending = s["block"].forward(s["ctx"], s["residual"], None, RUN)
    s["norm"].apply(s["residual"], pending, s["normed"])
    keys, values, _ = s["ctx"].cache.kv_of_entry(0)
    return {"normed": s["normed"], "stream": s["residual"], "keys": keys, "values": values}


def _latent_pass(s):
    return {"out": s["part"].forward(s["ctx"], s["x"], RUN), "pages": s["pages"]}


def _recurrent_pass(s):
    s["state"].zero_()                     # new requests: the engine zeroes a slot for its new occupant
    return {"out": s["part"].forward(s["ctx"], s["x"], RUN), "state": s["state"]}


def _experts_pass(s):
    return {"out": s["part"].forward(s["ctx"], s["x"])}


def run(state):
    k = state["kind"]
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if k == "sampling":
        return {"tokens": torch.tensor(state["sampler"].sample(state["logits"], state["params"], state["seeds"],
                                                               state["indices"], state["history"]))}
    if k.startswith("step"):
        eng = state["engine"]
        logits = eng.step(state["entries"])
        for e, start in zip(state["entries"], state["starts"]):      # the requests as they were, for the next pass
            eng.cache.truncate(e.slot, start)
        return {"logits": logits}
    if k == "layer_prompt":
        return _layer_pass(state)
    if k == "latent_prompt":
        return _latent_pass(state)
    if k == "experts":
        return _experts_pass(state)
    return _recurrent_pass(state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def work(case):
    k = case["kind"]
    if k == "sampling":
        return {"bytes": 4 * case["batch"] * case["vocab"], "flops": 0}
    if k == "experts":
        W, T = case["width"], case["tokens"]
        touched = EXPERTS * (1 - (1 - TOP / EXPERTS) ** T)
        per = 3 * W * (W // 2)
        return {"bytes": 2 * (touched * per + 3 * W * W + EXPERTS * W + 2 * T * W),
                "flops": 2 * T * (TOP * per + 3 * W * W + EXPERTS * W)}
    batch = _batch(case)
    T, held, pairs = sum(q for q, _ in batch), sum(s for _, s in batch), _pairs(batch)
    if k in ("layer_decode", "layer_prompt", "step_decode", "step_float32"):
        layers, hidden, heads, kv, hd, inter = _qwen(case)
        size = 4 if k == "step_float32" else 2
        per = hidden * hd * (2 * heads + 2 * kv) + 3 * hidden * inter
        out = {"bytes": layers * (size * per + size * 2 * kv * hd * (held + T)),
               "flops": layers * (2 * T * per + 4 * pairs * heads * hd)}
        if k.startswith("step"):
            vocab = case.get("vocab", VOCAB)
            out["bytes"] += size * vocab * hidden + 4 * len(batch) * vocab
            out["flops"] += 2 * len(batch) * vocab * hidden
        else:
            out["bytes"] += T * hidden * (2 + 4 + 2)            # the rows in; the stream and its normed form out
        return out
    W = case["width"]
    if k.startswith("latent"):
        H, dim, rot, dv, rank = _latent(case)
        per = W * (H * (dim + rot) + rank + rot + H + H * dv)
        up = H * (dim + dv) * rank
        own = 2 * pairs * H * (dim + rot + dv) + (2 * up * (T + held) if k == "latent_prompt" else 2 * up * T)
        if k == "latent_decode":                                # attended in the latent's space
            own = 2 * up * T + 2 * pairs * H * (2 * rank + rot)
        return {"bytes": 2 * (per + up) + 2 * (rank + rot) * (held + T) + 4 * T * W, "flops": 2 * T * per + own}
    if k == "delta_prompt":
        inner = W                                              # heads x 128
        per = W * (4 * inner + 2 * W // HEAD) + inner * W
        state = 4 * len(batch) * (inner * HEAD + 3 * inner * (TAPS - 1))
        return {"bytes": 2 * per + 4 * T * W + state, "flops": 2 * T * per + 6 * T * inner * HEAD}
    C, N, R, taps = _scan(case)
    per = 2 * C * W + C * (R + 2 * N) + C * R + C * W
    return {"bytes": 2 * per + 4 * T * W + 4 * len(batch) * C * (N + taps - 1), "flops": 2 * T * per + 6 * T * C * N}


def tolerance(case):
    k = case["kind"]
    if k == "sampling":
        return "exact"                     # whole numbers: token ids
    if k == "step_float32":
        return {"rel": 1e-5, "max": 4e-4}  # sums of 32-bit products in another order
    # activations and the cache rounded to 8 bits of mantissa between the kernels: a layer is 0.002 to 0.004 away from the
    # same in 64 bits, a stack of four 0.01
    return {"rel": 3e-2 if k == "step_decode" else 1.2e-2, "max": 0.4}


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------------

F = torch.float64


def _rms(x, w, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.to(F)


def _angles(positions, dims, base):
    i = torch.arange(dims // 2, dtype=F, device=DEV)
    a = positions.to(F)[:, None] * base ** (-2.0 * i / dims)
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _turn_halves(x, positions, base):
    c, s = _angles(positions, x.shape[-1], base)
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _turn_pairs(x, positions, base):
    c, s = _angles(positions, x.shape[-1], base)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)


def _attend(q, k, v, start, scale):
    """q [new, heads, d] behind ``start`` keys; k [keys, KV heads, d], v [keys, KV heads, dv]."""
    rep = q.shape[1] // k.shape[1]
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=F, device=DEV)
    mask = torch.arange(k.shape[0], device=DEV)[None] > (start + torch.arange(q.shape[0], device=DEV))[:, None]
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // rep].T) * scale
        out[:, h] = torch.softmax(s.masked_fill(mask, -math.inf), -1) @ v[:, h // rep]
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _qwen_layer(x, w, p, batch, cache, heads, kv, hd):
    lin = lambda a, n: a @ w[p + n].to(F).T
    n = _rms(x, w[p + "input_layernorm.weight"])
    T = x.shape[0]
    pos = torch.cat([torch.arange(s, s + q, device=DEV) for q, s in batch])
    q = _turn_halves(_rms(lin(n, "self_attn.q_proj.weight").view(T, heads, hd), w[p + "self_attn.q_norm.weight"]), pos, 1e6)
    k = _turn_halves(_rms(lin(n, "self_attn.k_proj.weight").view(T, kv, hd), w[p + "self_attn.k_norm.weight"]), pos, 1e6)
    v = lin(n, "self_attn.v_proj.weight").view(T, kv, hd)
    out, t, c = [], 0, 0
    for new, start in batch:
        kk = torch.cat([cache[0][c:c + start].to(F), k[t:t + new]])
        vv = torch.cat([cache[1][c:c + start].to(F), v[t:t + new]])
        out.append(_attend(q[t:t + new], kk, vv, start, hd ** -0.5))
        t, c = t + new, c + start
    x = x + lin(torch.cat(out).reshape(T, heads * hd), "self_attn.o_proj.weight")
    n = _rms(x, w[p + "post_attention_layernorm.weight"])
    return x + lin(_silu(lin(n, "mlp.gate_proj.weight")) * lin(n, "mlp.up_proj.weight"), "mlp.down_proj.weight")


def _causal_conv(x, taps_w):
    """y[t, c] = sum_j w[c, j] x[t - (taps - 1 - j), c], one request."""
    T, taps = x.shape[0], taps_w.shape[1]
    y = torch.zeros_like(x)
    for j in range(taps):
        back = taps - 1 - j
        if back < T:
            y[back:] += x[:T - back] * taps_w[:, j].to(F)
    return y


def exact(case, seed):
    k = case["kind"]
    if k == "sampling":
        return None
    inp = _inputs(case, seed)
    if k == "experts":
        w, x = inp["w"], inp["x"].to(F)
        lin = lambda a, n: a @ w["mlp." + n].to(F).T
        z = lin(x, "router") + w["mlp.router.b"].to(F)
        val, idx = z.topk(TOP, -1)
        share = torch.zeros_like(z).scatter(1, idx, torch.softmax(val, -1))

        def expert(a, e):
            g, u = lin(a, e + "gate").clamp(max=LIMIT), lin(a, e + "up").clamp(-LIMIT, LIMIT)
            return lin(g * torch.sigmoid(ALPHA * g) * (u + 1), e + "down")
        out = expert(x, "shared.")
        for e in range(EXPERTS):
            out += share[:, e:e + 1] * expert(x, "e%d." % e)
        return {"out": out}
    batch = _batch(case)
    if k in ("layer_decode", "layer_prompt", "step_decode", "step_float32"):
        layers, hidden, heads, kv, hd, inter = _qwen(case)
        w = inp["w"]
        x = w["model.embed_tokens.weight"][inp["ids"].long()].to(F)
        for i in range(layers):
            x = _qwen_layer(x, w, f"model.layers.{i}.", batch, inp["cache"][i], heads, kv, hd)
        if k.startswith("layer"):
            return {"normed": _rms(x, w["model.norm.weight"]), "stream": x, "keys": None, "values": None}
        last = torch.tensor([q for q, _ in batch], device=DEV).cumsum(0) - 1
        return {"logits": _rms(x[last], w["model.norm.weight"]) @ w["lm_head.weight"].to(F).T}
    w, x = inp["w"], inp["x"].to(F)
    lin = lambda a, n: a @ w["mix." + n].to(F).T
    T = x.shape[0]
    if k.startswith("latent"):
        H, dim, rot, dv, rank = _latent(case)
        pos = torch.cat([torch.arange(s, s + q, device=DEV) for q, s in batch])
        q = lin(x, "q").view(T, H, dim + rot)
        q = torch.cat([q[..., :dim], _turn_pairs(q[..., dim:], pos, 10000.0)], -1)
        kv = lin(x, "dkv")
        row = torch.cat([_rms(kv[:, :rank], w["mix.dkv.norm"]), _turn_pairs(kv[:, None, rank:], pos, 10000.0)[:, 0]], -1)
        out, t, c = [], 0, 0
        for new, start in batch:
            rows = torch.cat([inp["cache"][c:c + start].to(F), row[t:t + new]])
            n = rows.shape[0]
            keys = torch.cat([lin(rows[:, :rank], "uk").view(n, H, dim), rows[:, None, rank:].expand(n, H, rot)], -1)
            out.append(_attend(q[t:t + new], keys, lin(rows[:, :rank], "uv").view(n, H, dv), start, (dim + rot) ** -0.5))
            t, c = t + new, c + start
        o = torch.cat(out) * torch.sigmoid(lin(x, "g"))[:, :, None]
        return {"out": lin(o.reshape(T, H * dv), "o"), "pages": None}
    outs, t = [], 0
    for new, _ in batch:
        outs.append((_delta_exact if k == "delta_prompt" else _scan_exact)(case, w, x[t:t + new], lin))
        t += new
    return {"out": torch.cat(outs), "state": None}


def _delta_exact(case, w, x, lin):
    T, H = x.shape[0], case["width"] // HEAD
    part = lambda n: _silu(_causal_conv(lin(x, n), w["mix." + n + ".conv"])).view(T, H, HEAD)
    unit = lambda a: a / torch.sqrt((a * a).sum(-1, keepdim=True) + EPS)
    q, k, v = unit(part("q")) * HEAD ** -0.5, unit(part("k")), part("v")
    beta = torch.sigmoid(lin(x, "b"))
    decay = torch.exp(-torch.exp(w["mix.A_log"].to(F)) * torch.nn.functional.softplus(lin(x, "a") + w["mix.dt_bias"].to(F)))
    S = torch.zeros(H, HEAD, HEAD, dtype=F, device=DEV)
    o = torch.empty(T, H, HEAD, dtype=F, device=DEV)
    for t in range(T):
        S = S * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    o = _rms(o, w["mix.norm"]) * _silu(lin(x, "g")).view(T, H, HEAD)
    return lin(o.reshape(T, H * HEAD), "o")


def _scan_exact(case, w, x, lin):
    C, N, R, taps = _scan(case)
    xz = lin(x, "in")
    u, z = xz[:, :C], xz[:, C:]
    u = _silu(_causal_conv(u, w["mix.conv"]) + w["mix.conv.b"].to(F))
    dbc = lin(u, "x")
    dt = torch.nn.functional.softplus(lin(dbc[:, :R], "dt") + w["mix.dt.b"].to(F))
    A = -torch.exp(w["mix.A_log"].to(F))
    S = torch.zeros(C, N, dtype=F, device=DEV)
    y = torch.empty_like(u)
    for t in range(x.shape[0]):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * dbc[t, R:R + N]
        y[t] = S @ dbc[t, R + N:]
    return lin((y + w["mix.D"].to(F) * u) * _silu(z), "o")

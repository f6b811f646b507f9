"""What a user of the framework has it do, as cases that can be timed: whole decode steps through the step function, single
layers and single mixers and feed-forwards over prompt portions, in the sizes of the repository's own layouts and benchmark.

Kinds of case:

``decode``   a decode step of a Qwen3 model (a few of its layers, its whole vocabulary) through ``Runner.step``: what a server
             does all day.  One token per request; logits come back.  Batch 1 over a small model is where latency and launches
             count, long and ragged batches are where the cache's bytes count.
``layer``    one Qwen3 layer (norms, attention, gated feed-forward) over the tokens of a step: a whole prompt, or what a scheduler
             with a token budget mixes: portions of prompts behind what the cache holds beside requests that bring one token.
             ``float32``: the same in the engine's 32-bit mode, which `marin-run verify` runs.
``experts``  a routed feed-forward with a shared expert (Pununex): a prompt's tokens, or a decode batch's few.
``delta``    a gated delta rule behind short convolutions (Pununex) over prompts.
``pooled``   attention over a window and pooled blocks with mixed head weights (Vogunex) over a prompt.
``latent``   attention over a latent that keys and values share (Nirotar) over prompts.
``wkv``      time mixing with a decay that depends on the token (Lakulix) over prompts.

Sizes: the Qwen3-0.6B/4B/8B/14B layouts' widths and heads; the variants at the 4B layout's sizes, as ``bench.py --arch`` has them.
"""
import math
from types import SimpleNamespace

import torch

PAGE = 16
ROOM = 32            # decode: how many steps a sequence takes before it is set back to where it began
THETA = 1000000.0
EPS = 1e-6

#: hidden size, query heads, kv heads, feed-forward width, tied head
LAYOUTS = {"0.6b": (1024, 16, 8, 3072, True), "4b": (2560, 32, 8, 9728, True), "8b": (4096, 32, 8, 12288, False), "14b": (5120, 40, 8, 17408, False)}
HEAD = 128
VOCAB = 151936


def listed():
    return [
        # one user, a small model, a short conversation: the smallest call, bound by latency
        {"name": "decode one small", "kind": "decode", "layout": "0.6b", "layers": 8, "batch": 1, "context": 300, "ragged": False},
        # the benchmark's headline step (batch 8, context 4,096), four of the layers
        {"name": "decode eight", "kind": "decode", "layout": "4b", "layers": 4, "batch": 8, "context": 4096, "ragged": False},
        # a busy server: many requests of all lengths, a model with a head of its own
        {"name": "decode many ragged", "kind": "decode", "layout": "8b", "layers": 2, "batch": 61, "context": 3900, "ragged": True},
        # a prompt in one step, the benchmark's size
        {"name": "prompt layer", "kind": "layer", "layout": "4b", "dtype": "bfloat16", "portions": 1, "tokens": 2048, "cached": 0, "singles": 0},
        # a step under a token budget: portions of three prompts behind cached positions, beside requests that decode
        {"name": "mixed layer", "kind": "layer", "layout": "8b", "dtype": "bfloat16", "portions": 3, "tokens": 1171, "cached": 1500, "singles": 13},
        # the 32-bit mode over a prompt
        {"name": "float32 layer", "kind": "layer", "layout": "0.6b", "dtype": "float32", "portions": 1, "tokens": 333, "cached": 0, "singles": 0},
        # routed experts over a prompt and over a decode batch
        {"name": "experts prompt", "kind": "experts", "hidden": 2560, "ff": 3648, "experts": 8, "top": 2, "shared": 2432, "tokens": 2048},
        {"name": "experts few tokens", "kind": "experts", "hidden": 2560, "ff": 3648, "experts": 8, "top": 2, "shared": 2432, "tokens": 48},
        # recurrent mixers over prompts
        {"name": "delta rule prompts", "kind": "delta", "hidden": 2560, "heads": 20, "per_channel": True, "portions": 2, "tokens": 1900},
        {"name": "time mixing prompt", "kind": "wkv", "hidden": 2560, "heads": 40, "portions": 1, "tokens": 2048},
        # attention variants over prompts
        {"name": "pooled attention prompt", "kind": "pooled", "hidden": 2560, "window": 1024, "pool": 64, "portions": 1, "tokens": 2048},
        {"name": "latent attention prompts", "kind": "latent", "hidden": 2560, "portions": 3, "tokens": 2000},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "layer", "layer", "float32", "experts", "delta", "wkv", "pooled", "latent"])
    if kind == "decode":
        layout = rng.choice(["0.6b", "4b", "8b"])
        return {"kind": "decode", "layout": layout, "layers": {"0.6b": 8, "4b": 4, "8b": 2}[layout], "batch": _log(rng, 1, 64),
                "context": _log(rng, 200, 4096), "ragged": rng.random() < 0.6}
    if kind == "layer":
        portions = rng.randint(1, 4)
        return {"kind": "layer", "layout": rng.choice(["0.6b", "4b", "8b"]), "dtype": "bfloat16", "portions": portions,
                "tokens": _log(rng, 40 * portions, 2048), "cached": rng.choice([0, 0, rng.randint(20, 2000)]), "singles": rng.choice([0, 0, rng.randint(1, 24)])}
    if kind == "float32":
        return {"kind": "layer", "layout": rng.choice(["0.6b", "4b"]), "dtype": "float32", "portions": rng.randint(1, 2), "tokens": _log(rng, 16, 400),
                "cached": 0, "singles": 0}
    if kind == "experts":
        return {"kind": "experts", "hidden": rng.choice([2048, 2560]), "ff": 64 * rng.randint(20, 57), "experts": rng.choice([4, 8, 16]), "top": rng.randint(1, 2),
                "shared": 64 * rng.randint(16, 38), "tokens": _log(rng, 24, 2048)}
    portions = rng.randint(1, 4)
    tokens = _log(rng, 100 * portions, 2048)
    if kind == "delta":
        heads = rng.choice([16, 20])
        return {"kind": "delta", "hidden": 128 * heads, "heads": heads, "per_channel": rng.random() < 0.5, "portions": portions, "tokens": tokens}
    if kind == "wkv":
        heads = rng.choice([32, 40])
        return {"kind": "wkv", "hidden": 64 * heads, "heads": heads, "portions": portions, "tokens": tokens}
    if kind == "pooled":
        return {"kind": "pooled", "hidden": 2560, "window": rng.choice([512, 1024]), "pool": rng.choice([32, 64]), "portions": portions, "tokens": tokens}
    return {"kind": "latent", "hidden": rng.choice([2048, 2560]), "portions": portions, "tokens": tokens}


# ---- sizes -----------------------------------------------------------------------------------------------------------------

def _split(total, parts):
    """``total`` in ``parts`` uneven lengths."""
    weights = [2 * i + 3 for i in range(parts)]
    out = [total * w // sum(weights) for w in weights]
    out[-1] += total - sum(out)
    return out


def _entries(case):
    """What a step brings: per request (positions the cache holds, new tokens); requests with one token come first."""
    singles = case.get("singles", 0)
    cached = case.get("cached", 0)
    lens = _split(case["tokens"], case.get("portions", 1))
    first = [(cached + 1 + 37 * i % 256 if cached else 64 + 37 * i % 256, 1) for i in range(singles)]
    return first + [(cached * (i + 1) // len(lens), n) for i, n in enumerate(lens)]


def _contexts(case):
    """Decode: the length every request's sequence has when its first step begins."""
    out = []
    for i in range(case["batch"]):
        last = case["context"] if not case["ragged"] else max(48, case["context"] * (i + 1) // case["batch"])
        out.append(max(16, last - ROOM))
    return out


def _pairs(entries, window=None, pool=None):
    total = 0
    for cached, n in entries:
        for at in range(cached, cached + n):
            if window is None or at + 1 <= window:
                total += at + 1
            else:
                total += window + ((at - window + 1) // pool if pool else 0)
    return total


def _layer_sizes(layout):
    h, H, K, ff, _ = LAYOUTS[layout]
    return (H + 2 * K) * HEAD * h + h * H * HEAD + 3 * h * ff


def work(case):
    kind = case["kind"]
    if kind == "decode":
        h, H, K, ff, _ = LAYOUTS[case["layout"]]
        B, L = case["batch"], case["layers"]
        keys = sum(c + 1 for c in _contexts(case))
        weights = L * _layer_sizes(case["layout"]) + VOCAB * h
        return {"bytes": 2 * weights + L * keys * 4 * K * HEAD + B * VOCAB * 4 + B * h * 2, "flops": 2.0 * B * weights + 4.0 * L * keys * H * HEAD}
    if kind == "experts":
        T, h, ff, top, sh = case["tokens"], case["hidden"], case["ff"], case["top"], case["shared"]
        used = min(case["experts"], T * top)
        return {"bytes": 2 * (3 * h * ff * used + 3 * h * sh) + 4 * case["experts"] * h + T * h * (2 + 8),
                "flops": 2.0 * T * h * (3 * ff * top + 3 * sh + case["experts"])}
    entries = _entries(case)
    T = sum(n for _, n in entries)
    if kind == "layer":
        h, H, K, ff, _ = LAYOUTS[case["layout"]]
        size = 2 if case["dtype"] == "bfloat16" else 4
        weights = _layer_sizes(case["layout"])
        return {"bytes": size * weights + T * h * 8 + 2 * sum(c + n for c, n in entries) * K * HEAD * size,
                "flops": 2.0 * T * weights + 4.0 * _pairs(entries) * H * HEAD}
    h = case["hidden"]
    if kind == "delta":
        H = case["heads"]
        weights = 4 * h * H * 128 + h * H + (2 * (128 * h + H * 128 * 128) if case["per_channel"] else h * H + h * H * 128)
        return {"bytes": 2 * weights + T * h * (2 + 8) + 2 * case["portions"] * H * 128 * 128 * 4,
                "flops": 2.0 * T * weights + T * (8.0 * H * 128 * 128 + 2.0 * 3 * H * 128 * 4)}
    if kind == "wkv":
        H, n = case["heads"], 64 * case["heads"]
        weights = 5 * h * n + 64 * (h + n)
        return {"bytes": 2 * weights + T * h * (2 + 8) + 2 * case["portions"] * H * 64 * 64 * 4, "flops": 2.0 * T * weights + 6.0 * T * H * 64 * 64}
    if kind == "pooled":
        H, K = 32, 8
        weights = (2 * H + 2 * K) * HEAD * h
        pairs = _pairs(entries, case["window"], case["pool"])
        # every head's scores once, the heads' weights mixed, the mixed weights on the values of the head's own kv head
        return {"bytes": 2 * weights + T * h * (2 + 8) + T * K * HEAD * 4, "flops": 2.0 * T * weights + pairs * (4.0 * H * HEAD + 2.0 * H * H)}
    H = 32
    weights = h * H * 96 + h * 160 + 2 * H * 64 * 128 + h * H * 64
    return {"bytes": 2 * weights + T * h * (2 + 8) + T * 160 * 2, "flops": 2.0 * T * weights + 2.0 * _pairs(entries) * H * (160 + 128)}


def tolerance(case):
    # about four times the distance between the framework and ``exact`` (bf16 activations: 0.0015 of a layer's stream, 0.0017 of
    # routed experts', 0.0034 to 0.007 of a mixer's own output, 0.012 of logits behind eight layers; 32 bits: 7e-7)
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": {"decode": 0.03, "layer": 0.008, "experts": 0.008}.get(case["kind"], 0.02)}


# ---- inputs, made from the seed alone --------------------------------------------------------------------------------------------

class _Draws:
    def __init__(self, seed, dtype=torch.bfloat16):
        self.g, self.dtype = torch.Generator(device="cuda").manual_seed(int(seed)), dtype

    def normal(self, *shape, std=1.0, dtype=None):
        return (torch.randn(*shape, device="cuda", generator=self.g) * std).to(dtype or self.dtype)

    def matrix(self, rows, cols):
        return self.normal(rows, cols, std=cols ** -0.5)

    def norm(self, n):
        return 1.0 + 0.05 * torch.randn(n, device="cuda", generator=self.g)

    def small(self, *shape, std=0.02, mean=0.0):
        return mean + std * torch.randn(*shape, device="cuda", generator=self.g)

    def between(self, low, high, *shape):
        return low + (high - low) * torch.rand(*shape, device="cuda", generator=self.g)


def _qwen_layer(d, layout, prefix):
    h, H, K, ff, _ = LAYOUTS[layout]
    return {f"{prefix}.input_layernorm.weight": d.norm(h), f"{prefix}.self_attn.q_proj.weight": d.matrix(H * HEAD, h),
            f"{prefix}.self_attn.k_proj.weight": d.matrix(K * HEAD, h), f"{prefix}.self_attn.v_proj.weight": d.matrix(K * HEAD, h),
            f"{prefix}.self_attn.o_proj.weight": d.matrix(h, H * HEAD), f"{prefix}.self_attn.q_norm.weight": d.norm(HEAD),
            f"{prefix}.self_attn.k_norm.weight": d.norm(HEAD), f"{prefix}.post_attention_layernorm.weight": d.norm(h),
            f"{prefix}.mlp.gate_proj.weight": d.matrix(ff, h), f"{prefix}.mlp.up_proj.weight": d.matrix(ff, h), f"{prefix}.mlp.down_proj.weight": d.matrix(h, ff)}


def _inputs(case, seed):
    """The weights by name and the step's inputs: the same for ``prepare`` and for ``exact``."""
    kind = case["kind"]
    d = _Draws(seed, torch.float32 if case.get("dtype") == "float32" else torch.bfloat16)
    if kind == "decode":
        h, _, K, _, tied = LAYOUTS[case["layout"]]
        w = {"model.embed_tokens.weight": d.matrix(VOCAB, h), "model.norm.weight": d.norm(h)}
        if not tied:
            w["lm_head.weight"] = d.matrix(VOCAB, h)
        for n in range(case["layers"]):
            w.update(_qwen_layer(d, case["layout"], f"model.layers.{n}"))
        # what the cache holds, layer by layer and request by request: rotated keys and values
        kv = [[(d.normal(c, K, HEAD), d.normal(c, K, HEAD)) for c in _contexts(case)] for _ in range(case["layers"])]
        tokens = torch.randint(0, VOCAB, (case["batch"],), generator=torch.Generator().manual_seed(int(seed))).tolist()
        return w, kv, tokens
    if kind == "layer":
        h, _, K, _, _ = LAYOUTS[case["layout"]]
        w = _qwen_layer(d, case["layout"], "layer")
        kv = [(d.normal(c, K, HEAD), d.normal(c, K, HEAD)) for c, _ in _entries(case)]
        return w, kv, d.normal(sum(n for _, n in _entries(case)), h, dtype=torch.float32)
    h, T = case["hidden"], case["tokens"]
    if kind == "experts":
        ff, E, sh = case["ff"], case["experts"], case["shared"]
        w = {"mlp.router.weight": d.small(E, h, std=h ** -0.5), "mlp.router.correction": d.small(E)}
        for e in range(E):
            w.update({f"mlp.experts.{e}.gate_proj.weight": d.matrix(ff, h), f"mlp.experts.{e}.up_proj.weight": d.matrix(ff, h),
                      f"mlp.experts.{e}.down_proj.weight": d.matrix(h, ff)})
        w.update({"mlp.shared.gate_proj.weight": d.matrix(sh, h), "mlp.shared.up_proj.weight": d.matrix(sh, h), "mlp.shared.down_proj.weight": d.matrix(h, sh)})
        return w, None, d.normal(T, h)
    if kind == "delta":
        H = case["heads"]
        n = H * 128
        dt = torch.exp(d.between(math.log(1e-3), math.log(1e-1), n if case["per_channel"] else H))
        w = {"mix.dt_bias": torch.log(torch.expm1(dt)), "mix.A_log": torch.log(d.between(1.0, 16.0, H)), "mix.norm": d.norm(128), "mix.b": d.matrix(H, h),
             "mix.o": d.matrix(h, n)}
        for p in "qkv":
            w[f"mix.{p}"], w[f"mix.{p}.conv"] = d.matrix(n, h), d.small(n, 4, std=0.5)
        if case["per_channel"]:
            w.update({"mix.a1": d.matrix(128, h), "mix.a2": d.matrix(n, 128), "mix.g1": d.matrix(128, h), "mix.g2": d.matrix(n, 128)})
        else:
            w.update({"mix.a": d.matrix(H, h), "mix.g": d.matrix(n, h)})
        return w, None, d.normal(T, h)
    if kind == "wkv":
        n = 64 * case["heads"]
        w = {f"mix.mu.{s}": d.between(0.0, 1.0, h) for s in ("r", "k", "v", "g", "w")}
        w.update({f"mix.{p}": d.matrix(n, h) for p in "rkvg"})
        w.update({"mix.w1": d.matrix(64, h), "mix.w2": d.matrix(n, 64), "mix.w0": d.between(-6.0, -1.0, n), "mix.u": d.small(case["heads"], 64, std=0.5),
                  "mix.norm": d.norm(n), "mix.o": d.matrix(h, n)})
        return w, None, d.normal(T, h)
    if kind == "pooled":
        H, K = 32, 8
        w = {"mix.q_proj.weight": d.matrix(H * HEAD, h), "mix.k_proj.weight": d.matrix(K * HEAD, h), "mix.v_proj.weight": d.matrix(K * HEAD, h),
             "mix.o_proj.weight": d.matrix(h, H * HEAD), "mix.q_proj.bias": d.small(H * HEAD), "mix.k_proj.bias": d.small(K * HEAD),
             "mix.v_proj.bias": d.small(K * HEAD), "mix.talk": torch.eye(H, device="cuda") + d.small(H, H, std=0.05)}
        return w, None, d.normal(T, h)
    w = {"mix.q": d.matrix(32 * 96, h), "mix.dkv": d.matrix(160, h), "mix.dkv.norm": d.norm(128), "mix.uk": d.matrix(32 * 64, 128),
         "mix.uv": d.matrix(32 * 64, 128), "mix.o": d.matrix(h, 32 * 64), "mix.sink": d.small(32, std=0.5)}
    return w, None, d.normal(T, h)


# ---- through the framework ---------------------------------------------------------------------------------------------------------

def _position(spec):
    from marin_b200.parts import PartSpec

    return PartSpec(spec[0], spec[1])


def _part(case):
    """The mixer or feed-forward of a case, as its architecture builds it."""
    from marin_b200.parts import lookup

    kind = case["kind"]
    h = case["hidden"]
    if kind == "experts":
        return lookup("feedforward", "routed_experts")(
            name="mlp", hidden=h, intermediate=case["ff"], experts=case["experts"], top=case["top"], score="softmax", renormalize=True, weight_on="output",
            correction=True, groups=2, keep_groups=2, shared_intermediate=case["shared"])
    if kind == "delta":
        more = {"decay": "channel", "decay_rank": 128, "gate": "sigmoid", "gate_rank": 128} if case["per_channel"] else {"decay": "head", "gate": "silu"}
        return lookup("mixer", "delta_rule")(name="mix", hidden=h, heads=case["heads"], kv_heads=case["heads"], dim=128, vdim=128, taps=4, norm_eps=EPS, **more)
    if kind == "wkv":
        return lookup("mixer", "wkv")(name="mix", hidden=h, heads=case["heads"], dim=64, decay_rank=64, norm_eps=EPS)
    if kind == "pooled":
        return lookup("mixer", "pooled_attention")(
            name="mix", hidden=h, heads=32, kv_heads=8, head_dim=HEAD, v_head_dim=HEAD, scale=HEAD ** -0.5, bias=True, qk_norm=True, norm_eps=EPS,
            position=_position(("rope", {"head_dim": HEAD, "theta": 500000.0, "rotary_dim": 64})), window=case["window"], pool=case["pool"],
            softcap=50.0, talk=True)
    return lookup("mixer", "latent_attention")(
        name="mix", hidden=h, heads=32, head_dim=64, rot_dim=32, v_head_dim=64, kv_rank=128, scale=96 ** -0.5, norm_eps=EPS, sink="learned",
        position=_position(("rope", {"head_dim": 32, "theta": 500000.0, "rotary_dim": 32, "interleaved": True})))


def _qwen_block(layout):
    from marin_b200.parts import LayerSpec, PartSpec, lookup

    h, H, K, ff, _ = LAYOUTS[layout]
    mixer = PartSpec("gqa_attention", {"hidden": h, "heads": H, "kv_heads": K, "head_dim": HEAD, "qk_norm": True, "norm_eps": EPS, "window": None,
                                       "position": PartSpec("rope", {"head_dim": HEAD, "theta": THETA})})
    spec = LayerSpec(block="prenorm", norm=PartSpec("rmsnorm", {"dim": h, "eps": EPS}), mixer=mixer, feedforward=PartSpec("swiglu", {"hidden": h, "intermediate": ff}),
                     prefix="layer", names={"norm1": "input_layernorm", "mixer": "self_attn", "norm2": "post_attention_layernorm", "feedforward": "mlp"})
    return lookup("block", "prenorm")(spec)


def _put(k_pages, v_pages, table, k, v):
    """A request's keys and values ``[n, kv heads, head]`` into the pages its block table names."""
    n = k.shape[0]
    at = torch.arange(n, device=k.device)
    page = torch.as_tensor(table, device=k.device, dtype=torch.long)[at // PAGE]
    k_pages[page, :, at % PAGE] = k
    v_pages[page, :, at % PAGE] = v


def _decode_state(case, seed):
    from marin_b200.cache import CacheManager
    from marin_b200.config import Qwen3Config
    from marin_b200.engine import Runner, StepEntry, build_model
    from marin_b200.parts import Runtime

    h, H, K, ff, tied = LAYOUTS[case["layout"]]
    w, kv, tokens = _inputs(case, seed)
    model = build_model(Qwen3Config.from_dict({
        "architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": case["layers"], "hidden_size": h, "num_attention_heads": H,
        "num_key_value_heads": K, "head_dim": HEAD, "intermediate_size": ff, "vocab_size": VOCAB, "rope_theta": THETA, "rms_norm_eps": EPS,
        "tie_word_embeddings": tied, "max_position_embeddings": 8192}))
    rt = Runtime(torch.device("cuda:0"), torch.bfloat16)
    model.load(w, rt)
    lengths = _contexts(case)
    cache = CacheManager(model.cache_needs(), [e.cache_of for e in model.spec.schedule], PAGE, sum(-(-(c + ROOM + 1) // PAGE) for c in lengths), len(lengths))
    cache.allocate(rt.device, rt.dtype)
    runner = Runner(model, cache, rt, 4224)
    runner.enable_graphs([len(lengths)])
    entries = [StepEntry(i, [t], [0]) for i, t in enumerate(tokens)]
    state = SimpleNamespace(kind="decode", runner=runner, entries=entries, lengths=lengths, left=0)
    _rewind(state)
    runner.step(entries)                     # an engine that serves has captured its step long before
    for i in range(len(lengths)):
        runner.end(i)
    _rewind(state)
    for n, layer in enumerate(kv):
        for i, (k, v) in enumerate(layer):
            _put(cache.groups[0].k[n], cache.groups[0].v[n], cache.block_table(i, 0), k, v)
    return state


def _rewind(state):
    """Requests that begin anew at the lengths they had."""
    for i, c in enumerate(state.lengths):
        state.runner.begin(i)
        state.runner.cache.reserve(i, c)
        state.runner.cache.commit(i, c)
    state.left = ROOM


def prepare(case, seed):
    from marin_b200.cache import CacheManager
    from marin_b200.engine import Runner, StepEntry
    from marin_b200.parts import Runtime

    kind = case["kind"]
    if kind == "decode":
        return _decode_state(case, seed)
    rt = Runtime(torch.device("cuda:0"), torch.float32 if case.get("dtype") == "float32" else torch.bfloat16)
    w, kv, x = _inputs(case, seed)
    part = _qwen_block(case["layout"]) if kind == "layer" else _part(case)
    part.load(w, rt)
    assert not w, sorted(w)
    need = None if kind == "experts" else part.mixer.cache_need() if kind == "layer" else part.cache_need()
    entries = _entries(case)
    cache = CacheManager([need], [None], PAGE, sum(-(-(c + n) // PAGE) for c, n in entries), len(entries))
    cache.allocate(rt.device, rt.dtype)
    runner = Runner(SimpleNamespace(spec=SimpleNamespace(vocab_size=VOCAB)), cache, rt, 8192)
    for i, (c, n) in enumerate(entries):
        runner.begin(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, c + n)
    ctx = runner.build_context([StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(entries)])
    view = runner.views.view(0, ctx)
    if kind == "layer":
        for i, (k, v) in enumerate(kv):
            _put(view.k, view.v, cache.block_table(i, 0), k, v)
    stream = torch.zeros(x.shape, device=x.device, dtype=torch.float32)
    return SimpleNamespace(kind=kind, runner=runner, part=part, ctx=ctx, view=view, x=x, stream=stream, slots=[s.slot for s in ctx.spans])


def run(state):
    from marin_b200.kernels import ops

    if state.kind == "decode":
        if state.left == 0:
            for i in range(len(state.lengths)):
                state.runner.end(i)
            _rewind(state)
        state.left -= 1
        return {"logits": state.runner.step(state.entries)}
    state.ctx.extras.clear()                 # what a step's layers share is made anew in every step
    with ops.using(state.runner.scratch):
        if state.kind == "layer":
            state.stream.copy_(state.x)
            state.part.forward(state.stream, state.ctx, state.view)
            return {"stream": state.stream, "k": state.view.k, "v": state.view.v}
        state.stream.zero_()
        if state.kind == "experts":
            state.part.forward(state.x, state.ctx, state.stream)
            return {"stream": state.stream}
        state.part.forward(state.x, state.ctx, state.view, state.stream)
    if state.kind == "pooled":
        return {"stream": state.stream, "k": state.view.k, "v": state.view.v}
    if state.kind == "latent":
        return {"stream": state.stream, "rows": state.view.k}
    views = state.view if isinstance(state.view, tuple) else (state.view,)
    first, last = min(state.slots), max(state.slots)
    return {"stream": state.stream, "state": [v.state[first:last + 1] for v in views]}


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------------------------

def _rms(x, w=None, eps=EPS):
    y = x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _rotate(x, positions, theta, dims, neighbours=False):
    """``x`` [T, heads, n] turned over its first ``dims`` elements."""
    half = dims // 2
    angle = positions.double()[:, None] * theta ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / dims)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    out = x.clone()
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :half], x[..., half:dims])
    ra, rb = a * cos - b * sin, b * cos + a * sin
    if neighbours:
        out[..., 0:dims:2], out[..., 1:dims:2] = ra, rb
    else:
        out[..., :half], out[..., half:dims] = ra, rb
    return out


def _lin(x, w):
    return x @ w.double().t()


def _attend(q, k, v, first, scale):
    """Causal attention of queries [n, H, d] at positions first.. over keys and values [m, K, d]."""
    n, H, d = q.shape
    m, K, _ = k.shape
    out = torch.empty(n, H, v.shape[2], device=q.device, dtype=torch.float64)
    hide = torch.arange(m, device=q.device)[None, :] > first + torch.arange(n, device=q.device)[:, None]
    for j in range(K):
        heads = slice(j * (H // K), (j + 1) * (H // K))
        s = torch.einsum("nhd,md->hnm", q[:, heads], k[:, j]) * scale
        out[:, heads] = torch.einsum("hnm,md->nhd", s.masked_fill(hide, -math.inf).softmax(dim=-1), v[:, j])
    return out


def _qwen_exact(x, w, prefix, layout, entries, kv):
    h, H, K, ff, _ = LAYOUTS[layout]
    get = lambda name: w[f"{prefix}.{name}"]
    T = x.shape[0]
    positions = torch.cat([torch.arange(c, c + n, device=x.device) for c, n in entries])
    y = _rms(x, get("input_layernorm.weight"))
    q = _rotate(_rms(_lin(y, get("self_attn.q_proj.weight")).view(T, H, HEAD), get("self_attn.q_norm.weight")), positions, THETA, HEAD)
    k = _rotate(_rms(_lin(y, get("self_attn.k_proj.weight")).view(T, K, HEAD), get("self_attn.k_norm.weight")), positions, THETA, HEAD)
    v = _lin(y, get("self_attn.v_proj.weight")).view(T, K, HEAD)
    parts, at = [], 0
    for (c, n), (ck, cv) in zip(entries, kv):
        rows = slice(at, at + n)
        parts.append(_attend(q[rows], torch.cat([ck.double(), k[rows]]), torch.cat([cv.double(), v[rows]]), c, HEAD ** -0.5))
        at += n
    x = x + _lin(torch.cat(parts).reshape(T, H * HEAD), get("self_attn.o_proj.weight"))
    y = _rms(x, get("post_attention_layernorm.weight"))
    act = torch.nn.functional.silu(_lin(y, get("mlp.gate_proj.weight"))) * _lin(y, get("mlp.up_proj.weight"))
    return x + _lin(act, get("mlp.down_proj.weight"))


def _conv(x, w):
    """A causal convolution per channel: ``x`` [T, n], ``w`` [n, taps], the last column on the current token."""
    taps, T = w.shape[1], x.shape[0]
    pad = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(pad[j:j + T] * w[:, j].double() for j in range(taps))


def _delta_exact(x, w, case):
    H, T = case["heads"], x.shape[0]
    silu = torch.nn.functional.silu
    q, k, v = (silu(_conv(_lin(x, w[f"mix.{p}"]), w[f"mix.{p}.conv"])).view(T, H, 128) for p in "qkv")
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * 128 ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    beta = _lin(x, w["mix.b"]).sigmoid()
    if case["per_channel"]:
        a = (_lin(_lin(x, w["mix.a1"]), w["mix.a2"]) + w["mix.dt_bias"].double()).view(T, H, 128)
        gate = _lin(_lin(x, w["mix.g1"]), w["mix.g2"]).sigmoid()
    else:
        a = (_lin(x, w["mix.a"]) + w["mix.dt_bias"].double()).view(T, H, 1)
        gate = silu(_lin(x, w["mix.g"]))
    g = torch.exp(-w["mix.A_log"].double().exp()[None, :, None] * torch.nn.functional.softplus(a))
    S, o = x.new_zeros(H, 128, 128), x.new_empty(T, H, 128)
    for t in range(T):
        S = S * g[t, :, :, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        o[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return _lin((_rms(o, w["mix.norm"]).reshape(T, H * 128)) * gate, w["mix.o"]), S


def _wkv_exact(x, w, case):
    H, T = case["heads"], x.shape[0]
    before = torch.cat([x.new_zeros(1, x.shape[1]), x[:-1]])
    mix = {s: x + (before - x) * w[f"mix.mu.{s}"].double() for s in ("r", "k", "v", "g", "w")}
    r, k, v = (_lin(mix[p], w[f"mix.{p}"]).view(T, H, 64) for p in "rkv")
    gate = torch.nn.functional.silu(_lin(mix["g"], w["mix.g"]))
    decay = torch.exp(-torch.exp(_lin(_lin(mix["w"], w["mix.w1"]).tanh(), w["mix.w2"]) + w["mix.w0"].double())).view(T, H, 64)
    u = w["mix.u"].double()
    S, o = x.new_zeros(H, 64, 64), x.new_empty(T, H, 64)
    for t in range(T):
        kv = k[t, :, :, None] * v[t, :, None, :]
        o[t] = torch.einsum("hkv,hk->hv", S + u[:, :, None] * kv, r[t])
        S = S * decay[t, :, :, None] + kv
    return _lin((_rms(o).reshape(T, H * 64) * w["mix.norm"].double()) * gate, w["mix.o"]), torch.cat([S.reshape(-1), x[-1]])


def _pooled_exact(x, w, case):
    T, H, K, window, P = x.shape[0], 32, 8, case["window"], case["pool"]
    at = torch.arange(T, device=x.device)
    q, k, v = ((_lin(x, w[f"mix.{p}_proj.weight"]) + w[f"mix.{p}_proj.bias"].double()).view(T, -1, HEAD) for p in "qkv")
    q, k = (_rotate(_rms(t), at, 500000.0, 64) for t in (q, k))
    blocks = T // P
    kb, vb = (t[:blocks * P].view(blocks, P, K, HEAD).mean(dim=1) for t in (k, v))
    keys, values = torch.cat([k, kb]), torch.cat([v, vb])
    far = at[:, None] - at[None, :]
    seen = torch.cat([(far >= 0) & (far < window), (torch.arange(blocks, device=x.device) * P + P - 1)[None, :] <= at[:, None] - window], dim=1)
    out = x.new_empty(T, H, HEAD)
    for rows in torch.arange(T, device=x.device).split(256):
        s = torch.einsum("nkgd,mkd->kgnm", q[rows].view(-1, K, H // K, HEAD), keys).reshape(H, rows.numel(), -1) * HEAD ** -0.5
        p = (50.0 * torch.tanh(s / 50.0)).masked_fill(~seen[rows], -math.inf).softmax(dim=-1)
        p = torch.einsum("hg,gnm->hnm", w["mix.talk"].double(), p).view(K, H // K, rows.numel(), -1)
        out[rows] = torch.einsum("kgnm,mkd->nkgd", p, values).reshape(-1, H, HEAD)
    return _lin(out.reshape(T, H * HEAD), w["mix.o_proj.weight"])


def _latent_exact(x, w):
    T, H = x.shape[0], 32
    at = torch.arange(T, device=x.device)
    q = _lin(x, w["mix.q"]).view(T, H, 96)
    row = _lin(x, w["mix.dkv"])
    c = _rms(row[:, :128], w["mix.dkv.norm"])
    kr = _rotate(row[:, None, 128:], at, 500000.0, 32, True)
    qr = _rotate(q[..., 64:], at, 500000.0, 32, True)
    k, v = _lin(c, w["mix.uk"]).view(T, H, 64), _lin(c, w["mix.uv"]).view(T, H, 64)
    s = (torch.einsum("nhd,mhd->hnm", q[..., :64], k) + torch.einsum("nhd,md->hnm", qr, kr[:, 0])) * 96 ** -0.5
    s = s.masked_fill(at[None, :] > at[:, None], -math.inf)
    s = torch.cat([s, w["mix.sink"].double()[:, None, None].expand(H, T, 1)], dim=2).softmax(dim=-1)[..., :-1]
    return _lin(torch.einsum("hnm,mhd->nhd", s, v).reshape(T, H * 64), w["mix.o"])


def _experts_exact(x, w, case):
    silu = torch.nn.functional.silu
    glu = lambda y, p: _lin(silu(_lin(y, w[f"{p}.gate_proj.weight"])) * _lin(y, w[f"{p}.up_proj.weight"]), w[f"{p}.down_proj.weight"])
    scores = _lin(x, w["mlp.router.weight"]).softmax(dim=-1)
    chosen = (scores + w["mlp.router.correction"].double()).topk(case["top"], dim=-1).indices
    weights = scores.gather(1, chosen)
    weights = weights / weights.sum(dim=-1, keepdim=True)
    out = glu(x, "mlp.shared")
    for e in range(case["experts"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        out.index_add_(0, rows, glu(x[rows], f"mlp.experts.{e}") * weights[rows, place][:, None])
    return out


def exact(case, seed):
    w, kv, x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "decode":
        h = w["model.embed_tokens.weight"][torch.as_tensor(x, device="cuda")].double()
        entries = [(c, 1) for c in _contexts(case)]
        for n, layer in enumerate(kv):
            h = _qwen_exact(h, w, f"model.layers.{n}", case["layout"], entries, layer)
        head = w.get("lm_head.weight", w["model.embed_tokens.weight"])
        y = _rms(h, w["model.norm.weight"])
        return {"logits": torch.cat([_lin(y, rows) for rows in head.split(16384)], dim=1)}
    x = x.double()
    if kind == "layer":
        return {"stream": _qwen_exact(x, w, "layer", case["layout"], _entries(case), kv), "k": None, "v": None}
    if kind == "experts":
        return {"stream": _experts_exact(x, w, case)}
    parts = x.split(_split(case["tokens"], case["portions"]))
    if kind == "delta":
        got = [_delta_exact(p, w, case) for p in parts]
        return {"stream": torch.cat([g[0] for g in got]), "state": [torch.stack([g[1] for g in got]), None]}
    if kind == "wkv":
        got = [_wkv_exact(p, w, case) for p in parts]
        return {"stream": torch.cat([g[0] for g in got]), "state": [torch.stack([g[1] for g in got])]}
    if kind == "pooled":
        return {"stream": torch.cat([_pooled_exact(p, w, case) for p in parts]), "k": None, "v": None}
    return {"stream": torch.cat([_latent_exact(p, w) for p in parts]), "rows": None}

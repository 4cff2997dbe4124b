"""Cases for timing the engine: its layers and two whole models, at the sizes that serving meets.

Every layer is a part of the framework (``build_part``) stepped the way the decoder steps it: inputs, weights, cache
pages, state rows and the step's integer arrays are in hand, ``forward`` is timed.  The whole models go through
``ModelRunner.step``.  Sizes are those of the repository's benchmarks: Qwen2.5 1.5B, 7B and 14B layers, and the
designs at width 2,048 and 4,096 with heads of 128.  Prompts come whole, alone or several ragged ones in a step.

The kinds, and what each stands for:

feed_forward     the gated feed-forward of a decoder layer, from one decoded token to a whole prompt
attention        the Qwen2.5 attention layer over prompts: projections, rotation, cache write, attention
decode           a step of decoded tokens of a four-layer Qwen2.5 through the captured graph, logits out
prompt_f32       prompts through two float32 layers (the true 32-bit path) to logits
sample           temperature, top-k and top-p over the vocabulary, as the engine samples after a step
experts          routed experts over a prompt portion or a batch of decoded tokens (Bavetar, Malilorn forms)
masked           softmax attention with head norms, masks, bias, sink, gate (Gusorax, Mobunex, Tuterax forms)
latent           attention over one compressed latent a token (Bavetar, Mobunex forms)
delta            the gated delta rule behind short convolutions (Tuterax)
mixing           time mixing, a matrix state per head (Malilorn)
state_space      the selective state-space mixer (Bavetar)
pooled           window and pooled-block attention with mixed heads (Gebadra)
"""
import math

import torch

DEVICE = "cuda:0"
PAGE = 16
EPS = 1e-6
F64 = torch.float64

# hidden, intermediate, heads, key/value heads of the Qwen2.5 layers the benchmarks run
QWEN = {"1.5b": (1536, 8960, 12, 2), "7b": (3584, 18944, 28, 4), "14b": (5120, 13824, 40, 8)}
THETA = 1e6
VOCAB = 32000


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one user decoding: the smallest call, bound by the weights of one layer and by its launches
        dict(name="feed_forward_1_row", kind="feed_forward", rows=1, hidden=1536, inter=8960, act="silu"),
        # a 2,048-token prompt through the attention of a 7B layer
        dict(name="attention_2048", kind="attention", size="7b", lens="2048"),
        # the headline workload: batch 8 from 2,048-token contexts, layers of the 7B model
        dict(name="decode_8", kind="decode", size="7b", batch=8, context=2048),
        # three ragged prompts in one step of the 32-bit path, layers of the 1.5B model
        dict(name="prompt_f32", kind="prompt_f32", size="1.5b", lens="17,311,700"),
        # sampling after a step of 64 requests over the full vocabulary
        dict(name="sample_64", kind="sample", rows=64, vocab=152064, top_k=50, top_p=0.9),
        # a prompt through 32 experts of a quarter of the dense width
        dict(name="experts_2048", kind="experts", form="gated", rows=2048, hidden=2048, inter=1408, experts=32, top=4),
        # a prompt through the attention with turned values, capped scores and a learned sink
        dict(name="masked_2048", kind="masked", form="turned", lens="2048", hidden=2048, heads=16, dim=128, vdim=128),
        # a prompt through attention over latents
        dict(name="latent_2048", kind="latent", form="sink", lens="2048", hidden=2048, heads=16),
        # ragged prompts through a delta rule with a decay per channel
        dict(name="delta_ragged", kind="delta", form="channel", lens="1100,37,911", hidden=2048, heads=16, dim=128),
        # a prompt through time mixing
        dict(name="mixing_2048", kind="mixing", lens="2048", hidden=2048, heads=16, dim=128),
        # a prompt through the state-space mixer
        dict(name="state_space_2048", kind="state_space", lens="2048", hidden=2048, heads=64, state=128, groups=8),
        # a prompt through window and pooled-block attention
        dict(name="pooled_2048", kind="pooled", lens="2048", hidden=2048, heads=16, kv_heads=4, window=1024, pool=64),
    ]


def _spread(rng, low, high):
    """A whole number spread evenly over the logarithm of the range."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _lens(rng, low, high):
    """One to four prompts of ragged lengths, ``low`` to ``high`` tokens in all."""
    total = _spread(rng, low, high)
    n = min(rng.choice([1, 1, 2, 3, 4]), total)
    cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def draw(rng):
    kind = rng.choice(["feed_forward", "attention", "decode", "prompt_f32", "sample", "experts", "masked", "latent",
                       "delta", "mixing", "state_space", "pooled"])
    if kind == "feed_forward":
        hidden, inter = rng.choice([(1536, 8960), (2048, 5632), (3584, 18944), (4096, 11008), (5120, 13824)])
        return dict(kind=kind, rows=_spread(rng, 1, 1024), hidden=hidden, inter=inter,
                    act=rng.choice(["silu", "silu", "gelu_tanh"]))
    if kind == "attention":
        return dict(kind=kind, size=rng.choice(sorted(QWEN)), lens=_lens(rng, 48, 2048))
    if kind == "decode":
        batch = _spread(rng, 1, 16)
        return dict(kind=kind, size=rng.choice(["1.5b", "7b"]), batch=batch, context=_spread(rng, 200, 16384 // batch))
    if kind == "prompt_f32":
        return dict(kind=kind, size="1.5b", lens=_lens(rng, 16, 1028))
    if kind == "sample":
        return dict(kind=kind, rows=_spread(rng, 1, 64), vocab=rng.choice([32000, 151936, 152064]),
                    top_k=rng.choice([0, 20, 50]), top_p=rng.choice([0.8, 0.9, 1.0]))
    if kind == "experts":
        experts, top = rng.choice([(16, 2), (32, 4), (64, 4), (64, 6)])
        return dict(kind=kind, form=rng.choice(["gated", "squared"]), rows=_spread(rng, 8, 2048), hidden=2048,
                    inter=rng.choice([768, 1408]), experts=experts, top=top)
    if kind == "masked":
        dim, vdim = rng.choice([(128, 128), (128, 128), (64, 32)])
        return dict(kind=kind, form=rng.choice(["turned", "biased", "chunked", "unit"]), lens=_lens(rng, 48, 2048),
                    hidden=2048, heads=16, dim=dim, vdim=vdim)
    if kind == "latent":
        return dict(kind=kind, form=rng.choice(["sink", "stretched"]), lens=_lens(rng, 48, 2048), hidden=2048, heads=16)
    if kind == "delta":
        return dict(kind=kind, form=rng.choice(["channel", "head"]), lens=_lens(rng, 48, 2048), hidden=2048,
                    heads=rng.choice([8, 16]), dim=rng.choice([64, 128]))
    if kind == "mixing":
        return dict(kind=kind, lens=_lens(rng, 48, 2048), hidden=2048, heads=rng.choice([8, 16]),
                    dim=rng.choice([64, 128]))
    if kind == "state_space":
        return dict(kind=kind, lens=_lens(rng, 48, 2048), hidden=2048, heads=rng.choice([32, 64]),
                    state=rng.choice([64, 128]), groups=rng.choice([1, 8]))
    return dict(kind=kind, lens=_lens(rng, 48, 2048), hidden=2048, heads=16, kv_heads=rng.choice([2, 4]),
                window=rng.choice([256, 500, 1024]), pool=rng.choice([16, 64]))


# ------------------------------------------------------------------------------------------------ inputs
class _Random:
    """Tensors drawn one after the other on the GPU from one seed."""

    def __init__(self, seed, salt):
        self.gen = torch.Generator(device=DEVICE)
        self.gen.manual_seed(int(seed) * 64 + salt)

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device=DEVICE).normal_(mean, std, generator=self.gen)

    def uniform(self, shape, low, high):
        return torch.empty(shape, dtype=torch.float32, device=DEVICE).uniform_(low, high, generator=self.gen)

    def ints(self, shape, high):
        return torch.randint(0, high, shape, generator=self.gen, device=DEVICE)


def _matrices(r, shapes, dtype=torch.bfloat16, std=0.02):
    return {n: r.normal(s, std, dtype=dtype) for n, s in shapes.items()}


def _lengths(case):
    return [int(n) for n in case["lens"].split(",")]


def _rows(case):
    return int(case["rows"]) if "rows" in case else sum(_lengths(case))


def _step_sizes(r, n):
    """Biases whose softplus is spread over 0.001 to 0.1, as such models are set up."""
    return torch.log(torch.expm1(torch.exp(r.uniform((n,), math.log(1e-3), math.log(1e-1)))))


def _sizes(case):
    """(part category, kind, constants) of a layer case."""
    k, w = case["kind"], case.get("hidden")
    if k == "feed_forward":
        return "feed_forward", "swiglu", dict(hidden_size=w, intermediate_size=case["inter"], activation=case["act"])
    if k == "attention":
        w, _, heads, kv = QWEN[case["size"]]
        return "mixer", "attention", dict(hidden_size=w, num_heads=heads, num_kv_heads=kv, head_dim=128, qkv_bias=True,
                                          scale=128 ** -0.5, position=("rope", dict(theta=THETA, head_dim=128)))
    if k == "experts":
        a = dict(hidden_size=w, intermediate_size=case["inter"], num_experts=case["experts"], top=case["top"])
        if case["form"] == "gated":
            a.update(groups=4, keep=2, scale=2.5)
        else:
            a.update(router_score="sigmoid", normalize=False, weight_on="input", activation="relu2",
                     shared_size=case["inter"], shared_gate=True)
        return "feed_forward", "routed_experts", a
    if k == "masked":
        a = dict(hidden_size=w, num_heads=case["heads"], num_kv_heads=max(1, case["heads"] // 8), key_dim=case["dim"],
                 value_dim=case["vdim"], scale=case["dim"] ** -0.5, eps=EPS)
        a.update({"turned": dict(qk_norm=True, sink=True, softcap=30.0, rotate_values=True,
                                 rotary=dict(dims=case["dim"] // 2, base=1e6)),
                  "biased": dict(qk_norm=True, mask="window", mask_size=1024, distance_bias=dict(rows=32, far=1024.0)),
                  "chunked": dict(qk_norm=True, mask="chunk", mask_size=512, unit_sink=True, out_gate=True,
                                  proj_bias=True),
                  "unit": dict(qk_norm="unit", mask="window", mask_size=1024, proj_bias="qkv",
                               head_temperature=True)}[case["form"]])
        return "mixer", "masked_attention", a
    if k == "latent":
        a = dict(hidden_size=w, num_heads=case["heads"], head_dim=128, rot_dim=64, value_dim=128, kv_rank=512,
                 q_rank=w * 3 // 4, scale=192 ** -0.5, eps=EPS)
        if case["form"] == "sink":
            a.update(rotary=dict(base=1e6, dims=64), sink=True, out_gate=True)
        else:
            a.update(rotary=dict(base=1e6, dims=64, scaling=dict(factor=8.0, original=4096, fast=32.0, slow=1.0)),
                     sink=False, out_gate="each", window=1024)
        return "mixer", "latent_attention", a
    if k == "delta":
        channel = case["form"] == "channel"
        return "mixer", "gated_delta_rule", dict(
            hidden_size=w, num_heads=case["heads"], num_kv_heads=case["heads"] // 2, key_dim=case["dim"],
            value_dim=case["dim"], eps=EPS, conv_taps=4, decay=case["form"], gate="sigmoid" if channel else "silu",
            gate_low_rank=channel, unit_eps=1e-6)
    if k == "mixing":
        return "mixer", "time_mixing", dict(hidden_size=w, num_heads=case["heads"], key_dim=case["dim"], eps=EPS)
    if k == "state_space":
        return "mixer", "selective_state_space", dict(
            hidden_size=w, num_heads=case["heads"], head_dim=64, state_dim=case["state"], groups=case["groups"],
            conv_taps=4, norm_groups=8, eps=EPS)
    return "mixer", "pooled_window_attention", dict(
        hidden_size=w, num_heads=case["heads"], num_kv_heads=case["kv_heads"], key_dim=128, value_dim=128,
        scale=128 ** -0.5, window=case["window"], pool=case["pool"], eps=EPS,
        rotary=dict(base=500000.0, dims=64, factor=8.0),
        tensor_names=dict(q="q", k="k", v="v", o="o", q_norm="q.norm", k_norm="k.norm", talk="talk"), weight_suffix="")


def _layer_tensors(case, r):
    """The layer's checkpoint tensors by name."""
    k = case["kind"]
    a = _sizes(case)[2]
    w = a["hidden_size"]
    if k == "feed_forward":
        i = case["inter"]
        return _matrices(r, {"gate_proj.weight": (i, w), "up_proj.weight": (i, w), "down_proj.weight": (w, i)})
    if k == "attention":
        q, kv = a["num_heads"] * 128, a["num_kv_heads"] * 128
        t = _matrices(r, {"q_proj.weight": (q, w), "k_proj.weight": (kv, w), "v_proj.weight": (kv, w),
                          "o_proj.weight": (w, q)})
        t.update({n + "_proj.bias": r.normal((s,), 0.02) for n, s in (("q", q), ("k", kv), ("v", kv))})
        return t
    if k == "experts":
        i, E = case["inter"], case["experts"]
        t = _matrices(r, {"router": (E, w)})
        names = (["gate"] if case["form"] == "gated" else []) + ["up", "down"]
        for n in names:
            all_e = r.normal((E, w, i) if n == "down" else (E, i, w), 0.02, dtype=torch.bfloat16)
            t.update({f"e{e}.{n}": all_e[e] for e in range(E)})
        if case["form"] == "squared":
            t.update(_matrices(r, {"shared.up": (i, w), "shared.down": (w, i), "shared.sg": (1, w)}))
        return t
    if k == "masked":
        H, G, D, E = a["num_heads"], a["num_kv_heads"], a["key_dim"], a["value_dim"]
        t = _matrices(r, {"q": (H * D, w), "k": (G * D, w), "v": (G * E, w), "o": (w, H * E)})
        if case["form"] != "unit":
            t.update({"q.norm": r.normal((D,), 0.1, 1.0), "k.norm": r.normal((D,), 0.1, 1.0)})
        if case["form"] == "turned":
            t["sink"] = r.normal((H,))
        elif case["form"] == "biased":
            t["rel"] = r.normal((32, H), 0.5, dtype=torch.bfloat16)
        elif case["form"] == "chunked":
            t["g"] = r.normal((H * E, w), 0.02, dtype=torch.bfloat16)
            t.update({n + ".b": r.normal((s,), 0.02) for n, s in (("q", H * D), ("k", G * D), ("v", G * E), ("o", w))})
        else:
            t["temp"] = r.normal((H,), 0.1, 1.0)
            t.update({n + ".b": r.normal((s,), 0.02) for n, s in (("q", H * D), ("k", G * D), ("v", G * E))})
        return t
    if k == "latent":
        H, D, R, V, kv, qr = a["num_heads"], 128, 64, 128, 512, a["q_rank"]
        t = _matrices(r, {"dq": (qr, w), "uq": (H * (D + R), qr), "dkv": (kv + R, w), "uk": (H * D, kv),
                          "uv": (H * V, kv), "o": (w, H * V)})
        t.update({"dq.norm": r.normal((qr,), 0.1, 1.0), "dkv.norm": r.normal((kv,), 0.1, 1.0)})
        t["g"] = r.normal((H if case["form"] == "sink" else H * V, w), 0.02, dtype=torch.bfloat16)
        if case["form"] == "sink":
            t["sink"] = r.normal((H,))
        return t
    if k == "delta":
        H, G, D, E = a["num_heads"], a["num_kv_heads"], a["key_dim"], a["value_dim"]
        t = _matrices(r, {"q": (G * D, w), "k": (G * D, w), "v": (H * E, w), "b": (H, w), "o": (w, H * E)})
        t.update({n + ".conv": r.normal((s, 4), 0.3) for n, s in (("q", G * D), ("k", G * D), ("v", H * E))})
        t.update({"A_log": torch.log(r.uniform((H,), 1.0, 16.0)), "norm": r.normal((E,), 0.1, 1.0)})
        if case["form"] == "channel":
            t.update(_matrices(r, {"a1": (32, w), "a2": (H * D, 32), "g1": (32, w), "g2": (H * E, 32)}))
            t["dt_bias"] = _step_sizes(r, H * D)
        else:
            t.update(_matrices(r, {"a": (H, w), "g": (H * E, w)}))
            t["dt_bias"] = _step_sizes(r, H)
        return t
    if k == "mixing":
        n = a["num_heads"] * a["key_dim"]
        t = {"mu." + s: r.uniform((w,), 0.0, 1.0) for s in "rkvgw"}
        t.update(_matrices(r, {"r": (n, w), "k": (n, w), "v": (n, w), "g": (n, w), "w1": (32, w), "w2": (n, 32),
                               "o": (w, n)}))
        t.update({"w0": r.uniform((n,), -6.0, -1.0), "u": r.normal((a["num_heads"], a["key_dim"]), 0.3),
                  "norm": r.normal((n,), 0.1, 1.0)})
        return t
    if k == "state_space":
        H, inner, C = a["num_heads"], a["num_heads"] * 64, a["num_heads"] * 64 + 2 * a["groups"] * a["state_dim"]
        t = _matrices(r, {"in": (inner + C + H, w), "o": (w, inner)})
        t.update({"conv": r.normal((C, 4), 0.3), "conv.b": r.normal((C,), 0.02), "dt_bias": _step_sizes(r, H),
                  "A_log": torch.log(r.uniform((H,), 1.0, 16.0)), "D": r.normal((H,), 0.1, 1.0),
                  "norm": r.normal((inner,), 0.1, 1.0)})
        return t
    H, G, D = a["num_heads"], a["num_kv_heads"], 128
    t = _matrices(r, {"q": (H * D, w), "k": (G * D, w), "v": (G * D, w), "o": (w, H * D)})
    t.update({"q.norm": r.normal((H * D,), 0.1, 1.0), "k.norm": r.normal((G * D,), 0.1, 1.0),
              "talk": torch.eye(H, device=DEVICE) + r.normal((H, H), 0.1)})
    return t


def _layer_inputs(case, seed):
    r = _Random(seed, 1)
    tensors = _layer_tensors(case, r)
    return tensors, r.normal((_rows(case), _sizes(case)[2]["hidden_size"]), dtype=torch.bfloat16)


def _qwen_config(case):
    w, inter, heads, kv = QWEN[case["size"]]
    layers = 4 if case["kind"] == "decode" else 2
    return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=w, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=kv, head_dim=128, intermediate_size=inter,
                vocab_size=VOCAB, rope_theta=THETA, rms_norm_eps=EPS, tie_word_embeddings=False,
                max_position_embeddings=32768, use_sliding_window=False, hidden_act="silu", eos_token_id=VOCAB - 1)


def _qwen_inputs(case, seed):
    """(configuration, tensors by name, the requests' token ids)."""
    c, r = _qwen_config(case), _Random(seed, 2)
    dtype = torch.bfloat16 if case["kind"] == "decode" else torch.float32
    w, inter = c["hidden_size"], c["intermediate_size"]
    q, kv = c["num_attention_heads"] * 128, c["num_key_value_heads"] * 128
    t = _matrices(r, {"model.embed_tokens.weight": (VOCAB, w), "lm_head.weight": (VOCAB, w)}, dtype)
    t["model.norm.weight"] = r.normal((w,), 0.1, 1.0)
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        t.update(_matrices(r, {p + "self_attn.q_proj.weight": (q, w), p + "self_attn.k_proj.weight": (kv, w),
                               p + "self_attn.v_proj.weight": (kv, w), p + "self_attn.o_proj.weight": (w, q),
                               p + "mlp.gate_proj.weight": (inter, w), p + "mlp.up_proj.weight": (inter, w),
                               p + "mlp.down_proj.weight": (w, inter)}, dtype))
        t.update({p + f"self_attn.{n}_proj.bias": r.normal((s,), 0.02) for n, s in (("q", q), ("k", kv), ("v", kv))})
        t.update({p + n + ".weight": r.normal((w,), 0.1, 1.0) for n in ("input_layernorm", "post_attention_layernorm")})
    if case["kind"] == "decode":        # contexts of requests that arrived at different times, and the next token
        lens = [max(2, case["context"] - 13 * i) + 1 for i in range(case["batch"])]
    else:
        lens = _lengths(case)
    return c, t, [r.ints((n,), VOCAB).tolist() for n in lens]


def _wanted(case, n):
    """The places of a prompt whose logits are asked for: the last four, or fewer."""
    return list(range(max(0, n - 4), n))


# ------------------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "sample":
        from paged_batch_engine_b200 import SamplingParams
        from paged_batch_engine_b200.sampling.sampler import Sampler
        n = case["rows"]
        return dict(kind=kind, sampler=Sampler(torch.device(DEVICE), max_requests=n), counters=list(range(n)),
                    logits=_Random(seed, 3).normal((n, case["vocab"]), 2.5),
                    params=[SamplingParams(max_new_tokens=n + 1, temperature=0.8, top_k=case["top_k"],
                                           top_p=case["top_p"], seed=seed + i) for i in range(n)])
    from paged_batch_engine_b200.engine.batch import StepContext, StepEntry
    if kind in ("decode", "prompt_f32"):
        from paged_batch_engine_b200.engine.runner import ModelRunner, build_model
        config, tensors, requests = _qwen_inputs(case, seed)
        model = build_model(config, torch.bfloat16 if kind == "decode" else torch.float32, torch.device(DEVICE))
        model.build_kernels()
        model.load(tensors)
        longest = max(len(t) for t in requests)
        runner = ModelRunner(model, page_tokens=PAGE, max_requests=len(requests), max_context=longest + PAGE,
                             max_cache_tokens=sum(len(t) + 2 * PAGE for t in requests))
        entries = []
        for i, tokens in enumerate(requests):
            h = runner.cache.add_request(f"r{i}")
            if kind == "decode":
                assert runner.cache.reserve(h, len(tokens) - 1)
                runner.step([StepEntry(h, tokens[:-1])])
                tokens = tokens[-1:]
            assert runner.cache.reserve(h, len(tokens))
            entries.append(StepEntry(h, tokens, _wanted(case, len(tokens))))
        if kind == "decode":
            runner.step(entries, commit=False, decode_graph=True)       # the step's graph is captured once
        return dict(kind=kind, runner=runner, entries=entries, graph=kind == "decode")
    from paged_batch_engine_b200.cache.storage import CacheStorage
    from paged_batch_engine_b200.config import PartSpec
    from paged_batch_engine_b200.csrc.build import compile_many
    from paged_batch_engine_b200.parts import build_part
    category, name, args = _sizes(case)
    if "position" in args:
        args["position"] = PartSpec(*args["position"])
    part = build_part(category, PartSpec(name, args), torch.bfloat16, torch.device(DEVICE))
    compile_many(part.kernel_libraries(torch.bfloat16))
    tensors, x = _layer_inputs(case, seed)
    part.load(tensors, "")
    if category == "feed_forward":
        return dict(kind=kind, part=part, x=x, ctx=None)
    lens = _lengths(case)
    storage = CacheStorage([part.cache_need()], PAGE, sum(-(-n // PAGE) + 1 for n in lens), len(lens), torch.bfloat16,
                           torch.device(DEVICE))
    for held in storage.paged:
        for t in held.values():
            t.zero_()
    entries = []
    for i, n in enumerate(lens):
        h = storage.manager.add_request(f"r{i}")
        assert storage.manager.reserve(h, n)
        entries.append(StepEntry(h, [0] * n))
    cache = storage.layer(0)
    ctx = StepContext(storage.manager, entries, torch.device(DEVICE), part.paged_work(cache))
    return dict(kind=kind, part=part, x=x, ctx=ctx, cache=cache, states=list(storage.state.values()),
                pages=[t for held in storage.paged for t in held.values()])


def run(state):
    kind = state["kind"]
    if kind == "sample":
        return state["sampler"].sample_async(state["logits"], state["params"], state["counters"])[0]
    if "runner" in state:
        return state["runner"].step(state["entries"], commit=False, decode_graph=state["graph"])
    if state["ctx"] is None:
        return state["part"].forward(state["x"], None)
    for t in state["states"]:           # a request's state rows are zero when its first tokens run
        t.zero_()
    y = state["part"].forward(state["x"], state["ctx"], state["cache"])
    return dict(y=y, states=state["states"], pages=state["pages"])


# ------------------------------------------------------------------------------------------------ work
def _pairs(case, window=None):
    """Query-key pairs of causal attention over the case's prompts."""
    total = 0
    for n in _lengths(case):
        w = min(window or n, n)
        total += w * (w + 1) // 2 + (n - w) * w
    return total


def work(case):
    k = case["kind"]
    if k == "sample":
        return dict(bytes=4 * case["rows"] * (case["vocab"] + 1), flops=2 * case["rows"] * case["vocab"])
    if k in ("decode", "prompt_f32"):
        w, inter, heads, kv = QWEN[case["size"]]
        layers, size = (4, 2) if k == "decode" else (2, 4)
        layer = w * (2 * heads + 2 * kv) * 128 + 3 * w * inter
        if k == "decode":
            rows = wanted = case["batch"]
            pairs = sum(max(2, case["context"] - 13 * i) + 1 for i in range(rows))
            cached = pairs
        else:
            rows, wanted, pairs = _rows(case), sum(min(4, n) for n in _lengths(case)), _pairs(case)
            cached = rows
        return dict(bytes=size * (layers * (layer + 2 * kv * 128 * cached) + VOCAB * w + rows * w) + 4 * wanted * VOCAB,
                    flops=2 * rows * layers * layer + 4 * layers * heads * 128 * pairs + 2 * wanted * VOCAB * w)
    a, T = _sizes(case)[2], _rows(case)
    w = a["hidden_size"]
    if k == "feed_forward":
        m = 3 * w * case["inter"]
        return dict(bytes=2 * (m + 2 * T * w), flops=2 * T * m)
    if k == "experts":
        one = (3 if case["form"] == "gated" else 2) * w * case["inter"]
        E, top = case["experts"], case["top"]
        shared = one if case["form"] == "squared" else 0
        reached = E * (1.0 - (1.0 - top / E) ** T)          # experts that some row is expected to choose
        return dict(bytes=int(2 * (reached * one + shared + E * w + 2 * T * w)),
                    flops=2 * T * (top * one + shared + E * w))
    if k == "attention":
        H, G = a["num_heads"], a["num_kv_heads"]
        m = w * (2 * H + 2 * G) * 128
        return dict(bytes=2 * (m + 2 * T * w + 2 * T * G * 128), flops=2 * T * m + 4 * H * 128 * _pairs(case))
    if k == "masked":
        H, G, D, E = a["num_heads"], a["num_kv_heads"], a["key_dim"], a["value_dim"]
        m = w * (H * D + G * (D + E) + H * E + (H * E if case["form"] == "chunked" else 0))
        pairs = _pairs(case, a.get("mask_size"))
        if case["form"] == "chunked":
            pairs = sum((n // 512) * (512 * 513 // 2) + (n % 512) * (n % 512 + 1) // 2 for n in _lengths(case))
        return dict(bytes=2 * (m + 2 * T * w + T * G * (D + E)), flops=2 * T * m + 2 * H * (D + E) * pairs)
    if k == "latent":
        H, qr = a["num_heads"], a["q_rank"]
        m = w * (qr + 576) + qr * H * 192 + 2 * H * 128 * 512 + w * H * 128 + w * (H if case["form"] == "sink" else H * 128)
        return dict(bytes=2 * (m + 2 * T * w + T * 576), flops=2 * T * m + 2 * H * 320 * _pairs(case, a.get("window")))
    if k == "delta":
        H, G, D = a["num_heads"], a["num_kv_heads"], a["key_dim"]
        m = w * (2 * G * D + 2 * H * D + H) + (64 * (w + H * D) if case["form"] == "channel" else w * H * (D + 1))
        return dict(bytes=2 * (m + 2 * T * w) + 4 * len(_lengths(case)) * H * D * D, flops=2 * T * m + 6 * T * H * D * D)
    if k == "mixing":
        H, D = a["num_heads"], a["key_dim"]
        m = 5 * w * H * D + 32 * (w + H * D)
        return dict(bytes=2 * (m + 2 * T * w) + 4 * len(_lengths(case)) * H * D * D, flops=2 * T * m + 4 * T * H * D * D)
    if k == "state_space":
        H, N, G = a["num_heads"], a["state_dim"], a["groups"]
        m = w * (3 * H * 64 + 2 * G * N + H)
        return dict(bytes=2 * (m + 2 * T * w) + 4 * len(_lengths(case)) * H * N * 64, flops=2 * T * m + 4 * T * H * N * 64)
    H, G = a["num_heads"], a["num_kv_heads"]
    m = w * (2 * H + 2 * G) * 128
    pairs = _pairs(case, case["window"])
    pooled = sum(max(0, (p - case["window"] + 1) // case["pool"]) for n in _lengths(case) for p in range(n))
    return dict(bytes=2 * (m + 2 * T * w + 2 * T * G * 128),
                flops=2 * T * m + (4 * H * 128 + 2 * H * H) * (pairs + pooled))


def tolerance(case):
    k = case["kind"]
    if k == "sample":
        return "exact"
    if k == "prompt_f32":
        return {"rel": 1e-5}
    # four bf16 layers: 0.024 off the 64-bit logits, single layers 0.002 to 0.007
    return {"rel": 3e-2 if k == "decode" else 1e-2}


# ------------------------------------------------------------------------------------------------ 64-bit results
def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, pos, freq, back=False, pairs=False, dims=None):
    """x [T, heads, width]; the first ``dims`` values turned by position * freq, halves or neighbours paired."""
    dims = x.shape[-1] if dims is None else dims
    ang = (pos.to(F64)[:, None] * freq[None, :])[:, None, :] * (-1.0 if back else 1.0)
    c, s = torch.cos(ang), torch.sin(ang)
    out = x.clone()
    first = slice(0, dims, 2) if pairs else slice(0, dims // 2)
    second = slice(1, dims, 2) if pairs else slice(dims // 2, dims)
    a, b = x[..., first], x[..., second]
    out[..., first], out[..., second] = a * c - b * s, b * c + a * s
    return out


def _freq(dims, base):
    return float(base) ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEVICE) / dims)


def _causal(T, window=None, chunk=None):
    i = torch.arange(T, device=DEVICE)
    d = i[:, None] - i[None, :]
    see = d >= 0
    if window:
        see &= d < window
    if chunk:
        see &= (i // chunk)[:, None] == (i // chunk)[None, :]
    return see


def _attend(q, k, v, scale, see, cap=None, bias=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, E]; sink [H] or None."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=F64, device=DEVICE)
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].t() * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s + bias(h)
        s = s.masked_fill(~see, -math.inf)
        top = s.max(-1, keepdim=True).values
        if sink is not None:
            top = torch.clamp(top, min=float(sink[h]))
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink[h] - top)
        out[:, h] = (e / total) @ v[:, h // (H // G)]
    return out


def _conv(u, w, b=None):
    taps = w.shape[1]
    pad = torch.cat([torch.zeros((taps - 1, u.shape[1]), dtype=F64, device=DEVICE), u])
    y = sum(pad[j:j + u.shape[0]] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def _qwen_layer(x, w, p, c):
    T, H, G = x.shape[0], c["num_attention_heads"], c["num_key_value_heads"]
    h = _rms(x) * w[p + "input_layernorm.weight"]
    x = x + _gqa(h, {n[len(p + "self_attn."):]: t for n, t in w.items() if n.startswith(p + "self_attn.")}, H, G)
    h = _rms(x) * w[p + "post_attention_layernorm.weight"]
    return x + (_silu(h @ w[p + "mlp.gate_proj.weight"].t()) * (h @ w[p + "mlp.up_proj.weight"].t())) \
        @ w[p + "mlp.down_proj.weight"].t()


def _gqa(x, w, H, G):
    T = x.shape[0]
    pos, freq = torch.arange(T, device=DEVICE), _freq(128, THETA)
    q, k, v = (x @ w[n + "_proj.weight"].t() + w[n + "_proj.bias"] for n in "qkv")
    q, k = _turn(q.view(T, H, 128), pos, freq), _turn(k.view(T, G, 128), pos, freq)
    return _attend(q, k, v.view(T, G, 128), 128 ** -0.5, _causal(T)).reshape(T, H * 128) @ w["o_proj.weight"].t()


def _experts(x, w, case):
    E, top = case["experts"], case["top"]
    z = x @ w["router"].t()
    if case["form"] == "gated":
        s = torch.softmax(z, -1)
        best = s.view(-1, 4, E // 4).max(-1).values.topk(2, -1).indices
        kept = torch.zeros((x.shape[0], 4), dtype=torch.bool, device=DEVICE).scatter_(1, best, True)
        picked = s.masked_fill(~kept.repeat_interleave(E // 4, 1), -math.inf).topk(top, -1).indices
        g = s.gather(1, picked)
        g = g / g.sum(-1, keepdim=True) * 2.5
    else:
        picked = z.topk(top, -1).indices
        g = torch.sigmoid(z.gather(1, picked))
    out = torch.zeros_like(x)
    for e in range(E):
        row, place = torch.nonzero(picked == e, as_tuple=True)
        weight = g[row, place][:, None]
        if case["form"] == "gated":
            y = (_silu(x[row] @ w[f"e{e}.gate"].t()) * (x[row] @ w[f"e{e}.up"].t())) @ w[f"e{e}.down"].t() * weight
        else:
            y = torch.relu((x[row] * weight) @ w[f"e{e}.up"].t()) ** 2 @ w[f"e{e}.down"].t()
        out.index_add_(0, row, y)
    if case["form"] == "squared":
        shared = torch.relu(x @ w["shared.up"].t()) ** 2 @ w["shared.down"].t()
        out = out + shared * torch.sigmoid(x @ w["shared.sg"].t())
    return out


def _masked(x, w, a, form):
    H, G, D, E = a["num_heads"], a["num_kv_heads"], a["key_dim"], a["value_dim"]
    T = x.shape[0]
    pos = torch.arange(T, device=DEVICE)
    q, k, v = (x @ w[n].t() + (w[n + ".b"] if n + ".b" in w else 0.0) for n in "qkv")
    q, k, v = _rms(q.view(T, H, D)), _rms(k.view(T, G, D)), v.view(T, G, E)
    if form == "unit":
        q = q * w["temp"][:, None]
    else:
        q, k = q * w["q.norm"], k * w["k.norm"]
    if form == "turned":
        freq = _freq(D // 2, 1e6)
        q, k = _turn(q, pos, freq, dims=D // 2), _turn(k, pos, freq, dims=D // 2)
        v = _turn(v, pos, _freq(E, 1e6))
        o = _turn(_attend(q, k, v, a["scale"], _causal(T), cap=30.0, sink=w["sink"]), pos, _freq(E, 1e6), back=True)
    elif form == "biased":
        rows = [d if d < 16 else min(31, 16 + int(math.floor(math.log(d / 16) / math.log(1024.0 / 16) * 16)))
                for d in range(T)]
        d = (pos[:, None] - pos[None, :]).clamp(min=0)
        table = w["rel"][torch.tensor(rows, device=DEVICE)]
        o = _attend(q, k, v, a["scale"], _causal(T, window=1024), bias=lambda h: table[:, h][d])
    elif form == "chunked":
        sink = torch.zeros(H, dtype=F64, device=DEVICE)
        o = _attend(q, k, v, a["scale"], _causal(T, chunk=512), sink=sink)
    else:
        o = _attend(q, k, v, a["scale"], _causal(T, window=1024))
    o = o.reshape(T, H * E)
    if form == "chunked":
        return (o * torch.sigmoid(x @ w["g"].t())) @ w["o"].t() + w["o.b"]
    return o @ w["o"].t()


def _latent(x, w, a, form):
    H, T = a["num_heads"], x.shape[0]
    pos, freq, mag = torch.arange(T, device=DEVICE), _freq(64, 1e6), 1.0
    if form == "stretched":
        def dim_of(turns):
            return 64 * math.log(4096 / (2.0 * math.pi * turns)) / (2.0 * math.log(1e6))
        lo, hi = max(math.floor(dim_of(32.0)), 0), min(math.ceil(dim_of(1.0)), 63)
        ramp = ((torch.arange(32, dtype=F64, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        freq, mag = freq / 8.0 * ramp + freq * (1.0 - ramp), 0.1 * math.log(8.0) + 1.0
    q = ((_rms(x @ w["dq"].t()) * w["dq.norm"]) @ w["uq"].t()).view(T, H, 192)
    ckr = x @ w["dkv"].t()
    c = _rms(ckr[:, :512]) * w["dkv.norm"]
    qr = _turn(q[..., 128:], pos, freq, pairs=True) * mag
    kr = _turn(ckr[:, None, 512:], pos, freq, pairs=True) * mag
    k = torch.cat([(c @ w["uk"].t()).view(T, H, 128), kr.expand(T, H, 64)], -1)
    o = _attend(torch.cat([q[..., :128], qr], -1), k, (c @ w["uv"].t()).view(T, H, 128), a["scale"],
                _causal(T, window=a.get("window")), sink=w.get("sink"))
    gate = torch.sigmoid(x @ w["g"].t())
    o = o * gate[:, :, None] if form == "sink" else o * gate.view(T, H, 128)
    return o.reshape(T, H * 128) @ w["o"].t()


def _delta(x, w, a, form):
    H, G, D, T = a["num_heads"], a["num_kv_heads"], a["key_dim"], x.shape[0]
    q, k, v = (_silu(_conv(x @ w[n].t(), w[n + ".conv"])) for n in "qkv")

    def unit(y):
        y = y.view(T, G, D)
        return (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    q, k, v = unit(q) * D ** -0.5, unit(k), v.view(T, H, D)
    beta, rate = torch.sigmoid(x @ w["b"].t()), torch.exp(w["A_log"])
    if form == "channel":
        g = (x @ w["a1"].t() @ w["a2"].t() + w["dt_bias"]).view(T, H, D)
        g = torch.exp(-rate[:, None] * torch.nn.functional.softplus(g))
        gate = torch.sigmoid(x @ w["g1"].t() @ w["g2"].t())
    else:
        g = torch.exp(-rate * torch.nn.functional.softplus(x @ w["a"].t() + w["dt_bias"]))[:, :, None].expand(T, H, D)
        gate = _silu(x @ w["g"].t())
    S = torch.zeros((H, D, D), dtype=F64, device=DEVICE)
    o = torch.empty((T, H, D), dtype=F64, device=DEVICE)
    for t in range(T):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        o[t] = torch.einsum("hde,hd->he", S, q[t])
    return (_rms(o) * w["norm"] * gate.view(T, H, D)).reshape(T, H * D) @ w["o"].t(), S.transpose(1, 2)


def _mixing(x, w, a):
    H, D, T = a["num_heads"], a["key_dim"], x.shape[0]
    before = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
    blend = {s: x + (before - x) * w["mu." + s] for s in "rkvgw"}
    r, k, v, g = ((blend[s] @ w[s].t()).view(T, H, D) for s in "rkvg")
    decay = torch.exp(-torch.exp(w["w0"] + torch.tanh(blend["w"] @ w["w1"].t()) @ w["w2"].t())).view(T, H, D)
    bonus = (r * w["u"] * k).sum(-1, keepdim=True) * v
    S = torch.zeros((H, D, D), dtype=F64, device=DEVICE)
    o = torch.empty((T, H, D), dtype=F64, device=DEVICE)
    for t in range(T):
        o[t] = torch.einsum("hde,hd->he", S, r[t])
        S = S * decay[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
    y = _rms(o + bonus) * w["norm"].view(H, D) * _silu(g)
    return y.reshape(T, H * D) @ w["o"].t(), S.transpose(1, 2), x[-1]


def _state_space(x, w, a):
    H, N, G, T = a["num_heads"], a["state_dim"], a["groups"], x.shape[0]
    inner = H * 64
    proj = x @ w["in"].t()
    z, xbc, dt = proj[:, :inner], proj[:, inner:-H], torch.nn.functional.softplus(proj[:, -H:] + w["dt_bias"])
    xbc = _silu(_conv(xbc, w["conv"], w["conv.b"]))
    xs = xbc[:, :inner].view(T, H, 64)
    B, C = (xbc[:, inner + i * G * N:inner + (i + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    S = torch.zeros((H, N, 64), dtype=F64, device=DEVICE)
    y = torch.empty((T, H, 64), dtype=F64, device=DEVICE)
    for t in range(T):
        S = S * decay[t][:, None, None] + (dt[t][:, None] * B[t])[:, :, None] * xs[t][:, None, :]
        y[t] = torch.einsum("hnp,hn->hp", S, C[t])
    u = (y + w["D"][:, None] * xs).reshape(T, inner) * _silu(z)
    return (_rms(u.view(T, 8, inner // 8)).reshape(T, inner) * w["norm"]) @ w["o"].t(), S


def _pooled(x, w, a):
    H, G, T = a["num_heads"], a["num_kv_heads"], x.shape[0]
    window, pool = a["window"], a["pool"]
    pos, freq = torch.arange(T, device=DEVICE), _freq(64, 500000.0) / 8.0
    q, k = _rms(x @ w["q"].t()) * w["q.norm"], _rms(x @ w["k"].t()) * w["k.norm"]
    q, k = (_turn(y.view(T, n, 128), pos, freq, pairs=True, dims=64) for y, n in ((q, H), (k, G)))
    v = (x @ w["v"].t()).view(T, G, 128)
    n = T // pool
    keys = torch.cat([k, k[:n * pool].view(n, pool, G, 128).mean(1)])
    vals = torch.cat([v, v[:n * pool].view(n, pool, G, 128).mean(1)])
    blocks = torch.arange(n, device=DEVICE) * pool + pool - 1
    see = torch.cat([_causal(T, window=window), blocks[None, :] <= (pos - window)[:, None]], 1)
    o = torch.zeros((T, H, 128), dtype=F64, device=DEVICE)
    for h in range(H):          # o_h = sum over g of talk[h, g] * (softmax of head g) @ the values of head h
        s = (q[:, h] @ keys[:, h // (H // G)].t() * a["scale"]).masked_fill(~see, -math.inf)
        wts = torch.softmax(s, -1)
        for c in range(G):
            heads = slice(c * (H // G), (c + 1) * (H // G))
            o[:, heads] += w["talk"][heads, h][None, :, None] * (wts @ vals[:, c])[:, None, :]
    return o.reshape(T, H * 128) @ w["o"].t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None
    if kind in ("decode", "prompt_f32"):
        c, w, requests = _qwen_inputs(case, seed)
        w = {n: t.to(F64) for n, t in w.items()}
        rows = []
        for tokens in requests:
            x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEVICE)]
            for i in range(c["num_hidden_layers"]):
                x = _qwen_layer(x, w, f"model.layers.{i}.", c)
            x = x[-1:] if kind == "decode" else x[_wanted(case, len(tokens))]
            rows.append(_rms(x) * w["model.norm.weight"] @ w["lm_head.weight"].t())
        return torch.cat(rows)
    w, x = _layer_inputs(case, seed)
    w, x, a = {n: t.to(F64) for n, t in w.items()}, x.to(F64), _sizes(case)[2]
    if kind == "feed_forward":
        g = x @ w["gate_proj.weight"].t()
        g = _silu(g) if case["act"] == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
        return (g * (x @ w["up_proj.weight"].t())) @ w["down_proj.weight"].t()
    if kind == "experts":
        return _experts(x, w, case)
    ys, states, at = [], [], 0
    for n in _lengths(case):
        one = x[at:at + n]
        at += n
        if kind == "attention":
            y = _gqa(one, w, a["num_heads"], a["num_kv_heads"])
        elif kind == "masked":
            y = _masked(one, w, a, case["form"])
        elif kind == "latent":
            y = _latent(one, w, a, case["form"])
        elif kind == "pooled":
            y = _pooled(one, w, a)
        elif kind == "delta":
            y, *s = _delta(one, w, a, case["form"])
            states.append(s)
        elif kind == "mixing":
            y, *s = _mixing(one, w, a)
            states.append(s)
        else:
            y, *s = _state_space(one, w, a)
            states.append(s)
        ys.append(y)
    # the state rows lie in the order the requests came in, with one spare row behind them; what the
    # convolutions keep and the cache pages are not computed here
    rows = [torch.cat([torch.stack([s[j] for s in states]), torch.zeros_like(states[0][j])[None]])
            for j in range(len(states[0]))] if states else []
    if kind in ("delta", "state_space"):
        rows.append(None)
    pages = {"attention": 2, "masked": 2, "latent": 1, "pooled": 4}.get(kind, 0)
    return dict(y=torch.cat(ys), states=rows, pages=[None] * pages)

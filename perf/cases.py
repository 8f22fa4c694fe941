"""The work that a user of this library has it do, as cases that can be timed and compared.

Most cases are one sublayer of a model over a step's tokens, as a block runs it: the embedding's rows open the residual stream, the
norm's kernel reads them, the part works on the normed rows, and what it returns is added to the stream, which is the case's output
(with the recurrent parts' updated state records beside it).  Three cases are whole calls of `LLM.step`: prompts and then single tokens
through a model of a few layers, whose output is every step's logits.  Sizes are those of `bench.py` ("8b", "1b", "13b") and of its
designs' sizes "small", "lite" and "wide".

A case names its kind, its sizes, and `lens`, the tokens that each sequence of the step brings, joined by "+".  All inputs and
weights are drawn from the seed on the GPU."""

import math

import torch

DEV = "cuda:0"
PAGE = 64
VOCAB = 8192  # rows of the embedding that opens a sublayer's stream
EPS = 1e-5

LLAMA = {
    "1b": dict(d=2048, ff=5632, H=32, K=4, hd=64, vocab=32000, theta=10000.0, limit=2048, scaling=None),
    "8b": dict(d=4096, ff=14336, H=32, K=8, hd=128, vocab=128256, theta=500000.0, limit=131072, scaling={
        "rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}),
    "13b": dict(d=5120, ff=13824, H=40, K=40, hd=128, vocab=32000, theta=10000.0, limit=4096, scaling=None),
}
DESIGN = {
    "small": dict(d=1024, heads=8, dim=64, rot=32, vdim=64, rank=256, experts=16, top=2, eff=1024, sff=1024, hd=128, s_heads=32, s_groups=2),
    "lite": dict(d=2048, heads=16, dim=128, rot=64, vdim=128, rank=512, experts=64, top=6, eff=1408, sff=2816, hd=128, s_heads=64, s_groups=4),
    "wide": dict(d=4096, heads=32, dim=128, rot=64, vdim=128, rank=512, experts=32, top=4, eff=2048, sff=2048, hd=128, s_heads=128, s_groups=8),
}
STATE, S_VDIM, TAPS, DECAY_RANK, TAU = 128, 64, 4, 16, 8.0


def listed():
    return [
        # two prompts of unequal lengths through a grouped-query attention sublayer: the ordinary prompt step of the main model
        dict(name="attention_8b_prompts", kind="attention", size="8b", lens="1531+517", past=0),
        # the feed-forward of the same model over a prompt step: the largest products of the library
        dict(name="mlp_8b_prompt", kind="mlp", size="8b", lens="1777"),
        # routed experts with a shared one over a prompt step
        dict(name="experts_lite_prompt", kind="experts", size="lite", lens="2048"),
        # routed experts over few tokens (a large decode batch, short prompts): every expert's weights for a handful of rows
        dict(name="experts_wide_few", kind="experts", size="wide", lens="41+33+22"),
        # attention over cached latents, a prompt step of one sequence
        dict(name="latent_lite_prompt", kind="latent", size="lite", lens="2048"),
        # the same at small sizes with short prompts of very unequal lengths: little work, where launches count
        dict(name="latent_small_short", kind="latent", size="small", lens="300+41+5+222"),
        # gated linear attention over a prompt step
        dict(name="gla_lite_prompt", kind="gla", size="lite", lens="2048"),
        # the state-space layer over two prompts
        dict(name="ssm_lite_prompts", kind="ssm", size="lite", lens="1200+848"),
        # the gated delta rule behind short convolutions over three prompts
        dict(name="delta_lite_prompts", kind="delta", size="lite", lens="1029+700+319"),
        # a batch of 8 conversations: their prompts in one step, then 24 decode steps of the whole batch
        dict(name="serve_8b_batch8", kind="serve", size="8b", lens="96+33+64+7+128+71+50+80", layers=4, steps=24, dtype="bfloat16"),
        # one conversation on a small model: the smallest calls, one token a step
        dict(name="chat_1b_alone", kind="serve", size="1b", lens="45", layers=8, steps=48, dtype="bfloat16"),
        # a run in true 32-bit (what results are checked against): prompts and a few tokens
        dict(name="serve_1b_float32", kind="serve", size="1b", lens="219+64", layers=3, steps=12, dtype="float32"),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _cut(rng, total, most):
    """`total` tokens as up to `most` prompts of unequal lengths."""
    n = min(rng.randint(1, most), total)
    at = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return [b - a for a, b in zip([0] + at, at + [total])]


def draw(rng):
    kind = rng.choice(["attention", "mlp", "experts", "latent", "gla", "ssm", "delta", "serve"])
    join = lambda v: "+".join(str(n) for n in v)  # noqa: E731
    if kind in ("attention", "mlp"):
        size = rng.choice(["1b", "8b", "13b"])
        lens = _cut(rng, _spread(rng, 160, 1600 if size == "13b" else 2048), 4)
        case = dict(kind=kind, size=size, lens=join(lens))
        if kind == "attention":
            case["past"] = rng.choice([0, 0, rng.randint(1, 2048 - max(lens)) if max(lens) < 2048 else 0])
        return case
    if kind == "serve":
        if rng.random() < 0.25:
            return dict(kind=kind, size="1b", lens=join(_cut(rng, _spread(rng, 16, 280), 3)), layers=3, steps=rng.randint(4, 12), dtype="float32")
        size = rng.choice(["1b", "8b"])
        batch = _spread(rng, 1, 16)
        lens = [rng.randint(2, 128) for _ in range(batch)]
        return dict(kind=kind, size=size, lens=join(lens), layers=4, steps=rng.randint(8, 23 if size == "8b" else 48), dtype="bfloat16")
    size = rng.choice(["small", "lite", "wide"])
    if kind == "experts" and rng.random() < 0.4:
        return dict(kind=kind, size=size, lens=join(_cut(rng, _spread(rng, 9, 128), 6)))
    most = {"small": 3000, "lite": 2048, "wide": 1400}[size]
    return dict(kind=kind, size=size, lens=join(_cut(rng, _spread(rng, 130, most), 5)))


def _lens(case):
    return [int(n) for n in case["lens"].split("+")]


# ---------------------------------------------------------------------------------------------- inputs
class _Draw:
    """Numbers from the seed: the same for `prepare` and `exact`."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)

    def normal(self, shape, std, mean=0.0):
        return torch.randn(shape, generator=self.gen, dtype=torch.float32, device=DEV) * std + mean

    def uniform(self, shape, low, high):
        return torch.rand(shape, generator=self.gen, dtype=torch.float32, device=DEV) * (high - low) + low

    def matrix(self, rows, cols, gain=1.0, dtype=torch.bfloat16):
        return self.normal((rows, cols), gain / math.sqrt(cols)).to(dtype)

    def tokens(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.gen, dtype=torch.int32, device=DEV)


def _sublayer_weights(case, r):
    """The tensors of the sublayer's part, by their names in a checkpoint, in the types they are loaded in."""
    k = case["kind"]
    if k in ("attention", "mlp"):
        z = LLAMA[case["size"]]
        d = z["d"]
        if k == "mlp":
            return {"gate_proj.weight": r.matrix(z["ff"], d), "up_proj.weight": r.matrix(z["ff"], d), "down_proj.weight": r.matrix(d, z["ff"])}
        qd, kvd = z["H"] * z["hd"], z["K"] * z["hd"]
        return {"q_proj.weight": r.matrix(qd, d, 2.0), "k_proj.weight": r.matrix(kvd, d), "v_proj.weight": r.matrix(kvd, d), "o_proj.weight": r.matrix(d, qd)}
    z = DESIGN[case["size"]]
    d, H, hd = z["d"], z["heads"], z["hd"]
    if k == "experts":
        w = {}
        for i in range(z["experts"]):
            w[f"e{i}.gate"], w[f"e{i}.up"], w[f"e{i}.down"] = r.matrix(z["eff"], d), r.matrix(z["eff"], d), r.matrix(d, z["eff"])
        w["router"] = r.matrix(z["experts"], d).float()  # (a checkpoint stores the router's rows in bfloat16)
        w["shared.gate"], w["shared.up"], w["shared.down"] = r.matrix(z["sff"], d), r.matrix(z["sff"], d), r.matrix(d, z["sff"])
        return w
    if k == "latent":
        return {
            "q": r.matrix(H * (z["dim"] + z["rot"]), d, 2.0), "dkv": r.matrix(z["rank"] + z["rot"], d), "dkv.norm": r.normal((z["rank"],), 0.1, 1.0),
            "uk": r.matrix(H * z["dim"], z["rank"]), "uv": r.matrix(H * z["vdim"], z["rank"]), "sink": r.normal((H,), 0.5),
            "g": r.matrix(H * z["vdim"], d), "o": r.matrix(d, H * z["vdim"]),
        }
    if k == "gla":
        return {
            "q": r.matrix(H * hd, d), "k": r.matrix(H * hd, d), "v": r.matrix(H * hd, d), "g": r.matrix(H * hd, d), "a1": r.matrix(DECAY_RANK, d),
            "a2": r.matrix(H * hd, DECAY_RANK), "a2.b": r.normal((H * hd,), 0.5, 1.0), "norm": r.normal((hd,), 0.1, 1.0), "o": r.matrix(d, H * hd),
        }
    step = lambda n: r.uniform((n,), math.log(1e-3), math.log(1e-1)).exp().expm1().log()  # softplus of it is 0.001 to 0.1  # noqa: E731
    taps = lambda n: r.uniform((n, TAPS), -TAPS ** -0.5, TAPS ** -0.5)  # noqa: E731
    if k == "delta":
        return {
            "q": r.matrix(H * hd, d), "k": r.matrix(H * hd, d), "v": r.matrix(H * hd, d), "g": r.matrix(H * hd, d), "b": r.matrix(H, d), "a": r.matrix(H, d),
            "q.conv": taps(H * hd), "k.conv": taps(H * hd), "v.conv": taps(H * hd), "A_log": r.uniform((H,), 1.0, 16.0).log(), "dt_bias": step(H),
            "norm": r.normal((hd,), 0.1, 1.0), "o": r.matrix(d, H * hd),
        }
    SH, bc = z["s_heads"], z["s_groups"] * STATE
    inner = SH * S_VDIM
    return {
        "in": r.matrix(2 * inner + 2 * bc + SH, d), "conv": taps(inner + 2 * bc), "conv.b": r.normal((inner + 2 * bc,), 0.1), "dt_bias": step(SH),
        "A_log": r.uniform((SH,), 1.0, 16.0).log(), "D": r.normal((SH,), 0.1, 1.0), "norm": r.normal((inner,), 0.1, 1.0), "o": r.matrix(d, inner),
    }


def _width(case):
    return (LLAMA if case["size"] in LLAMA else DESIGN)[case["size"]]["d"]


def _sublayer_inputs(case, seed):
    r = _Draw(seed)
    d = _width(case)
    w = _sublayer_weights(case, r)
    table = r.normal((VOCAB, d), 1.0).to(torch.bfloat16)
    norm = r.normal((d,), 0.1, 1.0)
    lens = _lens(case)
    past = [r.tokens(case.get("past", 0), VOCAB) for _ in lens]
    return w, table, norm, past, [r.tokens(n, VOCAB) for n in lens]


def _llama_tensors(case, r):
    z, dt = LLAMA[case["size"]], getattr(torch, case["dtype"])
    d, qd, kvd = z["d"], z["H"] * z["hd"], z["K"] * z["hd"]
    w = {"model.embed_tokens.weight": r.normal((z["vocab"], d), 1.0).to(dt)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w[p + "self_attn.q_proj.weight"], w[p + "self_attn.k_proj.weight"] = r.matrix(qd, d, 2.0, dt), r.matrix(kvd, d, 1.0, dt)
        w[p + "self_attn.v_proj.weight"], w[p + "self_attn.o_proj.weight"] = r.matrix(kvd, d, 1.0, dt), r.matrix(d, qd, 1.0, dt)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"], w[p + "mlp.down_proj.weight"] = (
            r.matrix(z["ff"], d, 1.0, dt), r.matrix(z["ff"], d, 1.0, dt), r.matrix(d, z["ff"], 1.0, dt))
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = r.normal((d,), 0.1, 1.0).to(dt), r.normal((d,), 0.1, 1.0).to(dt)
    w["model.norm.weight"], w["lm_head.weight"] = r.normal((d,), 0.1, 1.0).to(dt), r.matrix(z["vocab"], d, 1.0, dt)
    return w


def _serve_inputs(case, seed):
    """The model's tensors, every sequence's prompt, and the tokens that each decode step brings."""
    r = _Draw(seed)
    w = _llama_tensors(case, r)
    vocab = LLAMA[case["size"]]["vocab"]
    prompts = [r.tokens(n, vocab).tolist() for n in _lens(case)]
    return w, prompts, [r.tokens(len(prompts), vocab).tolist() for _ in range(case["steps"])]


# ---------------------------------------------------------------------------------------------- the library's side
def _part(case, rt):
    from rusty_llama_b200.parts import FEED_FORWARDS, MIXERS
    from rusty_llama_b200.spec import PartSpec

    k = case["kind"]
    if k in ("attention", "mlp"):
        z = LLAMA[case["size"]]
        if k == "mlp":
            return FEED_FORWARDS.build(PartSpec("gated_mlp", {"hidden_size": z["d"], "intermediate_size": z["ff"], "activation": "silu"}), rt)
        pos = PartSpec("rotary", {"rotary_dim": z["hd"], "theta": z["theta"], "scaling": None, "interleaved": False})
        return MIXERS.build(PartSpec("attention", {"hidden_size": z["d"], "num_heads": z["H"], "num_kv_heads": z["K"], "head_dim": z["hd"], "window": 0, "position": pos}), rt)
    z = DESIGN[case["size"]]
    if k == "experts":
        return FEED_FORWARDS.build(PartSpec("routed_experts", {
            "hidden_size": z["d"], "n_experts": z["experts"], "top": z["top"], "expert_ff": z["eff"], "bias": False, "renormalize": True,
            "shared_ff": z["sff"], "shared_gate": False}), rt)
    if k == "latent":
        pos = PartSpec("rotary", {"rotary_dim": z["rot"], "theta": 10000.0, "scaling": None, "interleaved": False})
        return MIXERS.build(PartSpec("latent_attention", {
            "hidden_size": z["d"], "num_heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["rank"],
            "scale": 1.0 / math.sqrt(z["dim"] + z["rot"]), "eps": EPS, "position": pos}), rt)
    if k == "gla":
        return MIXERS.build(PartSpec("gated_linear_attention", {
            "hidden_size": z["d"], "num_heads": z["heads"], "dim": z["hd"], "vdim": z["hd"], "decay_rank": DECAY_RANK, "tau": TAU, "eps": EPS}), rt)
    if k == "delta":
        return MIXERS.build(PartSpec("gated_delta", {
            "hidden_size": z["d"], "num_heads": z["heads"], "num_qk_heads": z["heads"], "dim": z["hd"], "vdim": z["hd"], "taps": TAPS, "eps": EPS}), rt)
    return MIXERS.build(PartSpec("mamba2", {
        "hidden_size": z["d"], "num_heads": z["s_heads"], "vdim": S_VDIM, "state": STATE, "groups": z["s_groups"], "taps": TAPS,
        "norm_groups": z["s_groups"], "eps": EPS}), rt)


def _step(cache, slots, pos0, tokens):
    """The step's integers on the device, and the page tables of its sequences."""
    from rusty_llama_b200.engine import StepContext

    lens = [int(t.numel()) for t in tokens]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    tables, starts = [], [0]
    for n in lens:
        starts.append(starts[-1] + n)
    if cache is not None:
        cache.reserve(slots, lens)
        tables = [torch.from_numpy(cache.block_table(g, slots, cache.table_width(slots)).copy()).to(DEV) for g in range(len(cache.kv_groups))]
    ends = [p + n for p, n in zip(pos0, lens)]
    step = StepContext(
        n_tokens=sum(lens), n_seqs=len(lens), max_q_len=max(lens), max_kv_len=max(ends), plan_kv_len=max(ends), decode_only=max(lens) == 1,
        slots=list(slots), q_lens=lens, tokens=torch.cat(tokens), tok_seq=i32([i for i, n in enumerate(lens) for _ in range(n)]),
        tok_pos=i32([p + j for p, n in zip(pos0, lens) for j in range(n)]), seq_start=i32(starts), seq_pos0=i32(pos0), seq_len=i32(ends),
        slot_ids=i32(list(slots)), rows=None)
    return step, tables


def _prepare_sublayer(case, seed):
    from rusty_llama_b200.cache import Cache
    from rusty_llama_b200.parts import EMBEDDINGS, NORMS, Runtime
    from rusty_llama_b200.spec import PartSpec

    w, table, norm_w, past, tokens = _sublayer_inputs(case, seed)
    rt = Runtime.create(DEV, torch.bfloat16)
    d = _width(case)
    part = _part(case, rt)
    for p in (part,) + tuple(part.children()):
        p.load(w)
    embedding = EMBEDDINGS.build(PartSpec("token_embedding", {"vocab_size": VOCAB, "hidden_size": d}), rt)
    embedding.load({"weight": table})
    norm = NORMS.build(PartSpec("rmsnorm", {"size": d, "eps": EPS}), rt)
    norm.load({"weight": norm_w})
    s = dict(case=case, part=part, embedding=embedding, norm=norm, rt=rt, view=None, states=[])
    lens, n_past = _lens(case), case.get("past", 0)
    mixer = case["kind"] not in ("mlp", "experts")
    cache = None
    if mixer:
        pages = sum((n + n_past + PAGE - 1) // PAGE for n in lens)
        cache = Cache([(0, part.cache_need())], PAGE * pages, len(lens), torch.bfloat16, DEV)
    slots = [cache.open_sequence() for _ in lens] if mixer else list(range(len(lens)))
    if n_past:  # what the sequences hold already: an earlier portion of the same prompts
        s["step"], tables = _step(cache, slots, [0] * len(lens), past)
        s["view"] = cache.view(0, tables)
        _run_sublayer(s)
        cache.commit(slots, [n_past] * len(lens))
    s["step"], tables = _step(cache, slots, [n_past] * len(lens), tokens)
    if mixer:
        s["view"] = cache.view(0, tables)
        views = s["view"] if isinstance(s["view"], tuple) else (s["view"],)
        s["states"] = [v.state for v in views if hasattr(v, "state")]
    s["cache"] = cache
    return s


def _run_sublayer(s):
    stream = s["embedding"].forward(s["step"].tokens)
    xn = s["norm"].forward(stream)
    if s["view"] is None:
        stream.add(s["part"].forward(xn, s["step"]))
    else:
        for state in s["states"]:  # the sequences start here
            state.zero_()
        stream.add_result(s["part"].forward(xn, s["step"], s["view"]))
    stream.flush()
    return {"stream": stream.x, "states": s["states"]}


def _prepare_serve(case, seed):
    from rusty_llama_b200 import LLM
    from rusty_llama_b200.models.model import Model
    from rusty_llama_b200.parts import Runtime
    from rusty_llama_b200.registry import describe_model
    from rusty_llama_b200.weights.loader import load_tensors

    z = LLAMA[case["size"]]
    w, prompts, decode = _serve_inputs(case, seed)
    cfg = {
        "architectures": ["LlamaForCausalLM"], "tie_word_embeddings": False, "torch_dtype": case["dtype"], "hidden_size": z["d"],
        "intermediate_size": z["ff"], "num_hidden_layers": case["layers"], "num_attention_heads": z["H"], "num_key_value_heads": z["K"],
        "head_dim": z["hd"], "vocab_size": z["vocab"], "max_position_embeddings": z["limit"], "rms_norm_eps": EPS, "rope_theta": z["theta"],
        "rope_scaling": z["scaling"],
    }
    model = Model(describe_model(cfg), Runtime.create(DEV, case["dtype"]))
    load_tensors(model, w)
    torch.cuda.synchronize()
    llm = LLM(model, max_tokens=sum((len(p) + len(decode) + PAGE) // PAGE * PAGE for p in prompts), max_seqs=len(prompts))
    s = dict(case=case, llm=llm, prompts=prompts, decode=decode)
    _run_serve(s)  # a program's first requests: the decode step is captured
    return s


def _run_serve(s):
    from rusty_llama_b200 import StepEntry

    llm = s["llm"]
    slots = [llm.open_sequence() for _ in s["prompts"]]
    logits = [llm.step([StepEntry(slot, p, [len(p) - 1]) for slot, p in zip(slots, s["prompts"])])]
    for tokens in s["decode"]:
        logits.append(llm.step([StepEntry(slot, [t], [0]) for slot, t in zip(slots, tokens)]))
    for slot in slots:
        llm.close_sequence(slot)
    return logits


def prepare(case, seed):
    return _prepare_serve(case, seed) if case["kind"] == "serve" else _prepare_sublayer(case, seed)


def run(state):
    return _run_serve(state) if state["case"]["kind"] == "serve" else _run_sublayer(state)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    lens = _lens(case)
    T = sum(lens)
    if case["kind"] == "serve":
        z, L, S, D = LLAMA[case["size"]], case["layers"], len(lens), case["steps"]
        size = 2 if case["dtype"] == "bfloat16" else 4
        d, qd, kvd = z["d"], z["H"] * z["hd"], z["K"] * z["hd"]
        layer = d * (2 * qd + 2 * kvd) + 3 * d * z["ff"]
        weights = L * layer + d * z["vocab"]
        held = sum(n + t for n in lens for t in range(D))  # positions read by the decode steps
        pairs = sum(n * (n + 1) // 2 for n in lens) + sum(n + t + 1 for n in lens for t in range(D))
        nbytes = (D + 1) * (size * weights + 4 * S * z["vocab"]) + size * L * 2 * kvd * (held + T + S * D) + size * d * (T + S * D)
        flops = 2 * L * layer * (T + S * D) + 2 * d * z["vocab"] * S * (D + 1) + 4 * L * qd * pairs
        return {"bytes": nbytes, "flops": flops}
    d = _width(case)
    nbytes, flops = T * d * (2 + 4), 0  # the embedding's rows, the stream
    if case["kind"] == "mlp":
        n = 3 * d * LLAMA[case["size"]]["ff"]
        return {"bytes": nbytes + 2 * n, "flops": 2 * T * n}
    if case["kind"] == "attention":
        z, past = LLAMA[case["size"]], case.get("past", 0)
        qd, kvd = z["H"] * z["hd"], z["K"] * z["hd"]
        n = d * (2 * qd + 2 * kvd)
        pairs = sum(m * past + m * (m + 1) // 2 for m in lens)
        return {"bytes": nbytes + 2 * n + 2 * 2 * kvd * (T + past * len(lens)), "flops": 2 * T * n + 4 * qd * pairs}
    z = DESIGN[case["size"]]
    H, hd = z["heads"], z["hd"]
    if case["kind"] == "experts":
        used = z["experts"] * (1 - (1 - z["top"] / z["experts"]) ** T)  # experts that get a token
        expert, shared, router = 3 * d * z["eff"], 3 * d * z["sff"], d * z["experts"]
        return {"bytes": nbytes + 2 * (used * expert + shared) + 4 * router, "flops": 2 * T * (z["top"] * expert + shared + router)}
    if case["kind"] == "latent":
        # keys and values expanded from the latents once, or scores and sums taken in the latent space: the fewer operations
        n = d * (H * (z["dim"] + z["rot"]) + H * z["vdim"] * 2 + z["rank"] + z["rot"])
        up = H * (z["dim"] + z["vdim"]) * z["rank"]
        pairs = sum(m * (m + 1) // 2 for m in lens)
        inner = min(2 * H * pairs * (z["dim"] + z["rot"] + z["vdim"]), 2 * H * pairs * (2 * z["rank"] + z["rot"])) + 2 * T * up
        return {"bytes": nbytes + 2 * (n + up) + 2 * T * (z["rank"] + z["rot"]), "flops": 2 * T * n + inner}
    if case["kind"] in ("gla", "delta"):
        n = 5 * d * H * hd + (DECAY_RANK * (d + H * hd) if case["kind"] == "gla" else 2 * d * H)
        state = 4 * len(lens) * H * hd * hd
        return {"bytes": nbytes + 2 * n + state, "flops": 2 * T * n + (4 if case["kind"] == "gla" else 6) * T * H * hd * hd}
    SH = z["s_heads"]
    inner, bc = SH * S_VDIM, z["s_groups"] * STATE
    n = d * (3 * inner + 2 * bc + SH)
    return {"bytes": nbytes + 2 * n + 4 * len(lens) * SH * S_VDIM * STATE, "flops": 2 * T * n + 4 * T * SH * S_VDIM * STATE}


def tolerance(case):
    # about four times what the path was seen to be off the same in 64 bits: 0.0009 to 0.0019 for attention, latents and feed-forwards,
    # 0.0022 to 0.0048 for the recurrent parts and their states, 0.0075 (4 layers) to 0.011 (8 layers) for a model's logits, 2.8e-6 in 32-bit
    if case["kind"] == "serve":
        return {"rel": 1.2e-5 if case["dtype"] == "float32" else 2.5e-2}
    return {"rel": 1.5e-2 if case["kind"] in ("gla", "ssm", "delta") else 8e-3}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
F8 = torch.float64


def _rms(x, w, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.to(F8)


def _silu(x):
    return x * torch.sigmoid(x)


def _frequencies(n, theta, scaling=None):
    f = theta ** (-torch.arange(0, n, 2, dtype=F8, device=DEV) / n)
    if scaling is None:
        return f
    wave, old = 2 * math.pi / f, scaling["original_max_position_embeddings"]
    low, high, factor = scaling["low_freq_factor"], scaling["high_freq_factor"], scaling["factor"]
    smooth = ((old / wave - low) / (high - low)).clamp(0, 1)
    return (1 - smooth) * f / factor + smooth * f


def _turn(x, f, first=0):
    """x [T, heads, n]: pairs (j, j + n / 2) turned by position * f[j]."""
    angle = torch.arange(first, first + x.shape[0], dtype=F8, device=DEV)[:, None, None] * f
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def _attend(q, k, v, scale, sink=None):
    """q [T, H, n] at the last T of k's and v's [L, H, ...] positions."""
    out, L, T = [], k.shape[0], q.shape[0]
    seen = torch.arange(L, device=DEV)[None, :] <= torch.arange(L - T, L, device=DEV)[:, None]
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h].T * scale).masked_fill(~seen, -math.inf)
        if sink is None:
            p = torch.softmax(s, dim=-1)
        else:
            p = torch.softmax(torch.cat([s, sink[h].to(F8).expand(T, 1)], dim=1), dim=-1)[:, :-1]
        out.append(p @ v[:, h])
    return torch.stack(out, dim=1)


def _groups(x, n):
    return x.repeat_interleave(n, dim=1)


def _attention(z, w, xn, names, first):
    H, K, hd = z["H"], z["K"], z["hd"]
    f = _frequencies(hd, z["theta"], z["scaling"] if names is not None else None)
    g = lambda key: w[(names or "") + key + "_proj.weight"].to(F8)  # noqa: E731
    q, k, v = (xn[first:] @ g("q").T).view(-1, H, hd), (xn @ g("k").T).view(-1, K, hd), (xn @ g("v").T).view(-1, K, hd)
    o = _attend(_turn(q, f, first), _groups(_turn(k, f), H // K), _groups(v, H // K), hd ** -0.5)
    return o.flatten(1) @ g("o").T


def _latent(z, w, xn):
    H, dim, rot, vdim, rank = z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
    f = _frequencies(rot, 10000.0)
    q = (xn @ w["q"].to(F8).T).view(-1, H, dim + rot)
    raw = xn @ w["dkv"].to(F8).T
    c, kr = _rms(raw[:, :rank], w["dkv.norm"]), _turn(raw[:, None, rank:], f)
    k = torch.cat([(c @ w["uk"].to(F8).T).view(-1, H, dim), kr.expand(-1, H, -1)], dim=-1)
    v = (c @ w["uv"].to(F8).T).view(-1, H, vdim)
    q = torch.cat([q[..., :dim], _turn(q[..., dim:], f)], dim=-1)
    o = _attend(q, k, v, (dim + rot) ** -0.5, w["sink"]).flatten(1)
    return (o * torch.sigmoid(xn @ w["g"].to(F8).T)) @ w["o"].to(F8).T


def _recur(decay, k, v, q):
    """S <- diag(decay) S + k v^T, o = S^T q; decay [T, H, n or 1], k and q [T, H, n], v [T, H, m]."""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=F8, device=DEV)
    o = torch.empty_like(v)
    for t in range(k.shape[0]):
        S = S * decay[t, :, :, None] + k[t, :, :, None] * v[t, :, None, :]
        o[t] = torch.einsum("hnm,hn->hm", S, q[t])
    return o, S


def _gla(z, w, xn):
    H, hd = z["heads"], z["hd"]
    p = lambda key: (xn @ w[key].to(F8).T).view(-1, H, hd)  # noqa: E731
    a = torch.sigmoid((xn @ w["a1"].to(F8).T) @ w["a2"].to(F8).T + w["a2.b"].to(F8)).view(-1, H, hd) ** (1 / TAU)
    o, S = _recur(a, p("k"), p("v"), p("q") * hd ** -0.5)
    return (_rms(o, w["norm"]) * _silu(p("g"))).flatten(1) @ w["o"].to(F8).T, (S,)


def _conv(x, taps, bias=None):
    padded = torch.cat([torch.zeros(TAPS - 1, x.shape[1], dtype=F8, device=DEV), x])
    y = sum(padded[i : i + x.shape[0]] * taps[:, i].to(F8) for i in range(TAPS))
    return _silu(y if bias is None else y + bias.to(F8)), padded[x.shape[0] :]


def _delta(z, w, xn):
    H, hd = z["heads"], z["hd"]
    raw = torch.cat([xn @ w[key].to(F8).T for key in ("q", "k", "v")], dim=1)
    y, held = _conv(raw, torch.cat([w[key + ".conv"] for key in ("q", "k", "v")]))
    q, k, v = (t.view(-1, H, hd) for t in y.chunk(3, dim=1))
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * hd ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(xn @ w["b"].to(F8).T)
    g = torch.exp(-w["A_log"].to(F8).exp() * torch.nn.functional.softplus(xn @ w["a"].to(F8).T + w["dt_bias"].to(F8)))
    S, o = torch.zeros(H, hd, hd, dtype=F8, device=DEV), torch.empty_like(v)
    for t in range(xn.shape[0]):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hnm,hn->hm", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        o[t] = torch.einsum("hnm,hn->hm", S, q[t])
    gate = _silu((xn @ w["g"].to(F8).T).view(-1, H, hd))
    return (_rms(o, w["norm"]) * gate).flatten(1) @ w["o"].to(F8).T, (S, held)


def _ssm(z, w, xn):
    H, G = z["s_heads"], z["s_groups"]
    inner, bc = H * S_VDIM, G * STATE
    raw = xn @ w["in"].to(F8).T
    y, held = _conv(raw[:, inner : 2 * inner + 2 * bc], w["conv"], w["conv.b"])
    x = y[:, :inner].view(-1, H, S_VDIM)
    B, C = (_groups(t.reshape(-1, G, STATE), H // G) for t in (y[:, inner : inner + bc], y[:, inner + bc :]))
    dt = torch.nn.functional.softplus(raw[:, 2 * inner + 2 * bc :] + w["dt_bias"].to(F8))
    o, S = _recur(torch.exp(-w["A_log"].to(F8).exp() * dt)[:, :, None], B * dt[:, :, None], x, C)
    o = ((o + w["D"].to(F8)[:, None] * x).flatten(1) * _silu(raw[:, :inner])).view(-1, G, inner // G)
    return (o / torch.sqrt((o * o).mean(-1, keepdim=True) + EPS)).flatten(1) * w["norm"].to(F8) @ w["o"].to(F8).T, (S, held)


def _experts(z, w, xn):
    # chosen by the rows as the parts hand them on (bfloat16): a choice between two equal scores is not the path's to get right
    scores = torch.softmax(xn.to(torch.bfloat16).to(F8) @ w["router"].to(F8).T, dim=-1)
    weight, chosen = scores.topk(z["top"], dim=-1)
    weight = weight / weight.sum(-1, keepdim=True)
    mlp = lambda x, p: (_silu(x @ w[p + "gate"].to(F8).T) * (x @ w[p + "up"].to(F8).T)) @ w[p + "down"].to(F8).T  # noqa: E731
    y = mlp(xn, "shared.")
    for e in range(z["experts"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            y.index_add_(0, rows, mlp(xn[rows], f"e{e}.") * weight[rows, place, None])
    return y


def _exact_sublayer(case, seed):
    w, table, norm, past, tokens = _sublayer_inputs(case, seed)
    k = case["kind"]
    z = (LLAMA if case["size"] in LLAMA else DESIGN)[case["size"]]
    if k in ("mlp", "experts"):
        x = table[torch.cat(tokens).long()].to(F8)
        xn = _rms(x, norm)
        if k == "experts":
            return {"stream": x + _experts(z, w, xn), "states": []}
        h = _silu(xn @ w["gate_proj.weight"].to(F8).T) * (xn @ w["up_proj.weight"].to(F8).T)
        return {"stream": x + h @ w["down_proj.weight"].to(F8).T, "states": []}
    out, states = [], []
    for before, now in zip(past, tokens):
        x = table[torch.cat([before, now]).long()].to(F8)
        xn, n = _rms(x, norm), before.numel()
        if k == "attention":
            y, S = _attention(z, w, xn, None, n), ()
        elif k == "latent":
            y, S = _latent(z, w, xn), ()
        else:
            y, S = {"gla": _gla, "delta": _delta, "ssm": _ssm}[k](z, w, xn)
        out.append(x[n:] + y)
        states.append(S)
    # (slots are handed out in order, so record i is sequence i's)
    return {"stream": torch.cat(out), "states": [torch.stack(s) for s in zip(*states)]}


def _exact_serve(case, seed):
    w, prompts, decode = _serve_inputs(case, seed)
    z, D = LLAMA[case["size"]], case["steps"]
    rows = []
    for i, p in enumerate(prompts):
        tokens = torch.tensor(p + [step[i] for step in decode], device=DEV)
        x = w["model.embed_tokens.weight"][tokens].to(F8)
        for n in range(case["layers"]):
            name = f"model.layers.{n}."
            x = x + _attention(z, w, _rms(x, w[name + "input_layernorm.weight"]), name + "self_attn.", 0)
            h = _rms(x, w[name + "post_attention_layernorm.weight"])
            m = lambda key: w[name + "mlp." + key + "_proj.weight"].to(F8)  # noqa: E731, B023
            x = x + (_silu(h @ m("gate").T) * (h @ m("up").T)) @ m("down").T
        rows.append(_rms(x[len(p) - 1 :], w["model.norm.weight"]))
    head = w["lm_head.weight"].to(F8)
    return [torch.stack([r[t] for r in rows]) @ head.T for t in range(D + 1)]


def exact(case, seed):
    return _exact_serve(case, seed) if case["kind"] == "serve" else _exact_sublayer(case, seed)

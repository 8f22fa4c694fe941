"""The gated delta rule chunk by chunk against the recurrence in 64 bits and beside the token-by-token kernel: portions that are no
multiple of the chunk, sequences of one token beside long ones, several heads on one q/k head, sizes that leave tiles partly empty, decays
from none to ones that underflow inside a chunk, repeated keys; and the rule that takes a step there."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def recurrence(q, k, v, beta, decay, S):
    """One sequence in 64 bits: q, k [T, H, n], v [T, H, m], beta, decay [T, H], S [H, n, m]."""
    o = torch.empty(v.shape, dtype=torch.float64)
    for t in range(q.shape[0]):
        S = S * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hnm,hn->hm", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        o[t] = torch.einsum("hnm,hn->hm", S, q[t])
    return o, S


def inputs(lens, H, G, dim, vdim, seed, kind):
    g = torch.Generator().manual_seed(seed)
    T = sum(lens)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)  # noqa: E731
    q, k = unit(torch.randn(T, G, dim, generator=g)) * dim ** -0.5, unit(torch.randn(T, G, dim, generator=g))
    v = torch.randn(T, H, vdim, generator=g).to(torch.bfloat16)
    beta = torch.rand(T, H, generator=g)
    logd = -torch.rand(T, H, generator=g) * {"slow": 1e-3, "usual": 1.0, "fast": 60.0}.get(kind, 0.5)
    if kind == "repeated":  # the same few keys over and over, written at full strength: the system's entries are close to one
        k = k[torch.randint(0, 3, (T,), generator=g)]
        beta, logd = torch.ones(T, H), torch.zeros(T, H)
    return q, k, v, beta, logd


@pytest.mark.parametrize("kind", ["slow", "usual", "fast", "repeated"])
@pytest.mark.parametrize("lens, H, G, dim, vdim", [
    ([200, 64, 1, 63], 4, 2, 128, 128), ([65], 2, 2, 64, 20), ([130, 33], 3, 1, 36, 72), ([400], 2, 1, 100, 132), ([64, 128], 1, 1, 4, 4),
])
def test_against_64_bits_and_the_token_kernel(lens, H, G, dim, vdim, kind):
    from rusty_llama_b200.kernels import ops

    q, k, v, beta, logd = inputs(lens, H, G, dim, vdim, sum(lens) + dim, kind)
    T, S = sum(lens), len(lens)
    g = torch.Generator().manual_seed(1)
    start_state = torch.randn(S + 1, H, dim, vdim, generator=g)
    slots, starts = [S - i for i in range(S)], [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    wide = torch.zeros(T, H * vdim + 8, dtype=torch.bfloat16, device=DEV)
    wide[:, 8:] = v.view(T, -1).to(DEV)
    qd, kd = q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV)
    state, state1 = start_state.to(DEV), start_state.to(DEV)
    scratch = torch.full((ops.delta_chunked_scratch_floats(T, S, H, dim, vdim),), float("nan"), device=DEV)
    out = ops.delta_chunked(qd, kd, wide[:, 8:], beta.to(DEV), logd.to(DEV), state, i32(slots), i32(starts), H, G, dim, vdim, max(lens), scratch)
    one = ops.delta_rule(qd, kd, (q * k).sum(-1).contiguous().to(DEV), wide[:, 8:], beta.to(DEV), logd.exp().to(DEV), state1, i32(slots), i32(starts), H, G, dim, vdim)
    rep = H // G
    refs = [recurrence(*(t[a:b].double() for t in (q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1), v, beta, logd.exp().double())), start_state[slot].double())
            for a, b, slot in zip(starts, starts[1:], slots)]
    want, want_S = torch.cat([o for o, _ in refs]).reshape(T, -1), torch.stack([s for _, s in refs])
    rel = lambda x, y: float((x.double().cpu() - y).norm() / y.norm())  # noqa: E731
    # no worse than token by token (which rounds once a token), or a few roundings of 32 bits
    assert rel(out, want) <= max(1.5 * rel(one, want), 8 * 2.0 ** -24)
    assert rel(state[slots], want_S) <= max(1.5 * rel(state1[slots], want_S), 8 * 2.0 ** -24)
    assert torch.equal(state[0].cpu(), start_state[0])  # (nobody's record)


def test_which_steps_go_chunk_by_chunk():
    """A prompt of a bfloat16 run does, a short portion and a 32-bit run do not, and the layer's results agree within the run's rounding."""
    from rusty_llama_b200.cache import Cache
    from rusty_llama_b200.kernels import ops
    from rusty_llama_b200.parts import MIXERS, Runtime
    from rusty_llama_b200.spec import PartSpec

    from test_parts import ctx_for

    part = MIXERS.build(PartSpec("gated_delta", {"hidden_size": 64, "num_heads": 2, "num_qk_heads": 1, "dim": 32, "vdim": 48, "taps": 4, "eps": 1e-5}), Runtime.create(DEV, torch.bfloat16))
    g = torch.Generator().manual_seed(0)
    w = {}
    for name, info in part.param_infos().items():
        t = torch.randn(info.shape, generator=g) * (0.2 if len(info.shape) > 1 else 0.5) + (1.0 if name == "norm" else 0.0)
        w[name] = (t if info.kind == "scalars" else t.to(torch.bfloat16)).to(DEV)
    part.load(w)
    x = torch.randn(150, 64, generator=g).to(torch.bfloat16).to(DEV)
    called, before = [], ops.delta_chunked
    ops.delta_chunked = lambda *a, **k: called.append(1) or before(*a, **k)
    try:
        outs = []
        for cuts in ([150], [100, 31, 19], [31] * 4 + [26]):
            cache = Cache([(0, part.cache_need())], 64, 1, torch.bfloat16, DEV)
            slot, at, parts = cache.open_sequence(), 0, []
            for n in cuts:
                step, tables = ctx_for(cache, [slot], [at], [n])
                y = part.forward(x[at : at + n], step, cache.view(0, tables))
                parts.append(y.float().sum(0) if y.dim() == 3 else y.float())
                cache.commit([slot], [n])
                at += n
            outs.append((torch.cat(parts), len(called)))
    finally:
        ops.delta_chunked = before
    assert [n for _, n in outs] == [1, 2, 2]
    for y, _ in outs[1:]:
        assert float((y - outs[0][0]).norm() / outs[0][0].norm()) < 1e-2


@pytest.mark.parametrize("dim, vdim", [(128, 128), (36, 72)])
def test_decays_of_zero(dim, vdim):
    """A log decay of minus infinity (or far below what an exponential of 32 bits can hold) empties the state and the tokens after it go on
    from there, inside a chunk, at its first and last token and several times over."""
    from rusty_llama_b200.kernels import ops

    lens, H, G = [200, 64], 2, 1
    q, k, v, beta, logd = inputs(lens, H, G, dim, vdim, 5, "usual")
    for t, h, value in ((5, 0, float("-inf")), (6, 0, float("-inf")), (63, 0, float("-inf")), (64, 1, float("-inf")), (130, 1, -1e30), (200, 0, float("-inf")), (263, 1, -3e38)):
        logd[t, h] = value
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    T = sum(lens)
    state = torch.randn(2, H, dim, vdim, generator=torch.Generator().manual_seed(2))
    sd = state.to(DEV)
    scratch = torch.empty(ops.delta_chunked_scratch_floats(T, 2, H, dim, vdim), device=DEV)
    out = ops.delta_chunked(q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV), v.view(T, -1).to(DEV), beta.to(DEV), logd.to(DEV), sd, i32([0, 1]), i32([0, 200, 264]),
                            H, G, dim, vdim, max(lens), scratch)
    rep = H // G
    refs = [recurrence(*(t[a:b].double() for t in (q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1), v, beta, logd.double().exp())), state[i].double())
            for i, (a, b) in enumerate(((0, 200), (200, 264)))]
    want, want_S = torch.cat([o for o, _ in refs]).reshape(T, -1), torch.stack([s for _, s in refs])
    assert float((out.double().cpu() - want).norm() / want.norm()) <= 32 * 2.0 ** -24
    assert float((sd.double().cpu() - want_S).norm() / want_S.norm()) <= 32 * 2.0 ** -24


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_what_is_no_number_does_not_reach_earlier_tokens(value):
    """A value that is infinite or no number spoils its head's outputs from its token on and the state, and nothing before it."""
    from rusty_llama_b200.kernels import ops

    T, H, n = 150, 2, 64
    q, k, v, beta, logd = inputs([T], H, 1, n, n, 8, "usual")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    scratch = torch.empty(ops.delta_chunked_scratch_floats(T, 1, H, n, n), device=DEV)

    def run(v):
        state = torch.zeros(1, H, n, n, device=DEV)
        out = ops.delta_chunked(q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV), v.reshape(T, -1).to(DEV), beta.to(DEV), logd.to(DEV), state, i32([0]), i32([0, T]),
                                H, 1, n, n, T, scratch)
        return out.view(T, H, n), state[0]

    want, want_S = run(v)
    for at in (0, 1, 17, 63, 64, 149):
        bad = v.clone()
        bad[at, 0] = value
        out, S = run(bad)
        assert torch.equal(out[:at], want[:at]) and torch.equal(out[:, 1], want[:, 1]) and torch.equal(S[1], want_S[1]), at
        assert not bool(out[at:, 0].isfinite().any()) and not bool(S[0].isfinite().any())


def layer(H, G, dim, vdim, d):
    from rusty_llama_b200.parts import MIXERS, Runtime
    from rusty_llama_b200.spec import PartSpec

    part = MIXERS.build(PartSpec("gated_delta", {"hidden_size": d, "num_heads": H, "num_qk_heads": G, "dim": dim, "vdim": vdim, "taps": 4, "eps": 1e-5}),
                        Runtime.create(DEV, torch.bfloat16))
    g = torch.Generator().manual_seed(0)
    w = {}
    for name, info in part.param_infos().items():
        t = torch.randn(info.shape, generator=g) * (0.2 if len(info.shape) > 1 else 0.5) + (1.0 if name == "norm" else 0.0)
        w[name] = (t if info.kind == "scalars" else t.to(torch.bfloat16)).to(DEV)
    part.load(w)
    return part


def test_prompts_of_rising_lengths_leave_no_scratch_behind():
    from rusty_llama_b200.cache import Cache

    from test_parts import ctx_for

    part = layer(8, 2, 64, 64, 64)
    cache = Cache([(0, part.cache_need())], 64, 1, torch.bfloat16, DEV)
    slot = cache.open_sequence()

    def held(n):
        step, tables = ctx_for(cache, [slot], [0], [n])
        part.forward(torch.zeros(n, 64, dtype=torch.bfloat16, device=DEV), step, cache.view(0, tables))
        del step, tables
        torch.cuda.synchronize()
        return torch.cuda.memory_allocated()

    first = held(64)
    assert [held(n) - first for n in (128, 256, 512, 1024, 64)] == [0] * 5


def test_a_prompt_without_room_for_the_chunks_goes_token_by_token():
    from rusty_llama_b200.cache import Cache

    from test_parts import ctx_for
    from test_waits import with_memory_left

    part = layer(32, 1, 128, 128, 64)
    x = torch.randn(1024, 64, generator=torch.Generator().manual_seed(6)).to(torch.bfloat16).to(DEV)

    def run():
        cache = Cache([(0, part.cache_need())], 64, 1, torch.bfloat16, DEV)
        step, tables = ctx_for(cache, [cache.open_sequence()], [0], [1024])
        y = part.forward(x, step, cache.view(0, tables))
        return y.float().sum(0) if y.dim() == 3 else y.float()

    scratch = 4 * (1024 // 64 + 2) * 32 * (64 * 256 + 128 * 128 + 68)
    got = with_memory_left(scratch, run)  # (the rest of the layer takes some 60 MB of these 75)
    want = run()
    assert float((got - want).norm() / want.norm()) < 1e-2


def test_a_short_sequence_gets_the_token_kernels_bits_beside_a_prompt():
    """Which kernel takes a sequence's tokens depends on its own length: beside a prompt a single token and a short portion keep the bits
    that they have alone."""
    from rusty_llama_b200.cache import Cache
    from rusty_llama_b200.kernels import ops

    from test_parts import ctx_for

    part = layer(4, 2, 32, 48, 64)
    lens = [1, 100, 31, 64, 5]
    cache = Cache([(0, part.cache_need())], 64, len(lens), torch.bfloat16, DEV)
    slots = [cache.open_sequence() for _ in lens]
    x = torch.randn(sum(lens), 64, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).to(DEV)
    step, tables = ctx_for(cache, slots, [0] * len(lens), lens)
    view = cache.view(0, tables)
    records = next(v.state for v in (view if isinstance(view, tuple) else (view,)) if v.state.dim() == 4)
    records.normal_(generator=torch.Generator(device=DEV).manual_seed(3))
    start, seen = records.clone(), {}
    spied = {name: getattr(ops, name) for name in ("delta_prep", "short_conv", "head_norm_gate")}

    def spy(name):
        def call(*a, **k):
            seen[name] = (a, k, spied[name](*a, **k))
            return seen[name][2]
        return call

    try:
        for name in spied:
            setattr(ops, name, spy(name))
        part.forward(x, step, view)
    finally:
        for name, f in spied.items():
            setattr(ops, name, f)
    a, k, _ = seen["delta_prep"]
    qn, kn, kq, beta, decay = spied["delta_prep"](*a, **dict(k, log_decay=False))
    alone = ops.delta_rule(qn, kn, kq, seen["short_conv"][2][:, 2 * part.qd :], beta, decay, start, step.slot_ids, step.seq_start, 4, 2, 32, 48)
    o, at = seen["head_norm_gate"][0][0], 0
    for i, n in enumerate(lens):
        same = torch.equal(o[at : at + n], alone[at : at + n]) and torch.equal(records[slots[i]], start[slots[i]])
        if n < 32:
            assert same, f"{n} tokens"
        else:
            assert float((o[at : at + n] - alone[at : at + n]).norm() / alone[at : at + n].norm()) < 1e-5
        at += n


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("what", ["k", "beta", "logd"])
def test_what_is_no_number_does_not_reach_earlier_tokens_from_elsewhere(what, value):
    """The same for a token's key, its strength and its decay (one that grows without bound is no number either)."""
    from rusty_llama_b200.kernels import ops

    T, H, n = 150, 2, 64
    q, k, v, beta, logd = inputs([T], H, 2, n, n, 9, "usual")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    scratch = torch.empty(ops.delta_chunked_scratch_floats(T, 1, H, n, n), device=DEV)

    def run(k, beta, logd):
        state = torch.zeros(1, H, n, n, device=DEV)
        out = ops.delta_chunked(q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV), v.reshape(T, -1).to(DEV), beta.to(DEV), logd.to(DEV), state, i32([0]), i32([0, T]),
                                H, 2, n, n, T, scratch)
        return out.view(T, H, n), state[0]

    want, want_S = run(k, beta, logd)
    for at in (0, 1, 17, 63, 64, 149):
        bad = {"k": k.clone(), "beta": beta.clone(), "logd": logd.clone()}
        if what == "k":
            bad["k"][at, 0, 5] = value
        else:
            bad[what][at, 0] = value
        out, S = run(**bad)
        assert torch.equal(out[:at], want[:at]) and torch.equal(out[:, 1], want[:, 1]) and torch.equal(S[1], want_S[1]), at
        assert not bool(out[at:, 0].isfinite().any()) and not bool(S[0].isfinite().any()), at


@pytest.mark.parametrize("dim, vdim", [(128, 128), (36, 72), (64, 20)])
def test_the_norm_taken_along(dim, vdim):
    """The same sums through the norm inside the last kernel and behind it: a rounding of each of two 32-bit chains apart, then rounded to
    bfloat16 (2^-8 at most where that falls on different sides); wider values than a block has columns for are left to the caller."""
    from rusty_llama_b200.kernels import ops

    lens, H, G = [130, 40], 2, 1
    q, k, v, beta, logd = inputs(lens, H, G, dim, vdim, 11, "usual")
    T, g = sum(lens), torch.Generator().manual_seed(3)
    gate, w = torch.randn(T, H * vdim, generator=g).to(torch.bfloat16).to(DEV), torch.randn(vdim, generator=g).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    scratch = torch.empty(ops.delta_chunked_scratch_floats(T, 2, H, dim, vdim), device=DEV)

    def run(norm):
        return ops.delta_chunked(q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV), v.reshape(T, -1).to(DEV), beta.to(DEV), logd.to(DEV),
                                 torch.zeros(2, H, dim, vdim, device=DEV), i32([0, 1]), i32([0, 130, 170]), H, G, dim, vdim, 130, scratch, norm=norm)

    got = run((w, 1e-5, gate, ops.GATE_SILU, 0.5, None))
    want = ops.head_norm_gate(run(None), H, vdim, w, 1e-5, gate, ops.GATE_SILU, torch.bfloat16, out_scale=0.5)
    assert got.dtype == torch.bfloat16 and float(((got.float() - want.float()).abs() / (want.float().abs() + 1e-3)).max()) <= 2.0 ** -7
    assert float((got != want).float().mean()) <= 0.01
    assert run((w, 1e-5, gate, ops.GATE_SILU, 0.5, torch.empty(T, H * vdim + 1, dtype=torch.bfloat16, device=DEV)[:, 1:])) is None


def _layer(seed=0):
    from rusty_llama_b200.parts import MIXERS, Runtime
    from rusty_llama_b200.spec import PartSpec

    part = MIXERS.build(PartSpec("gated_delta", {"hidden_size": 64, "num_heads": 4, "num_qk_heads": 2, "dim": 32, "vdim": 48, "taps": 4, "eps": 1e-5}), Runtime.create(DEV, torch.bfloat16))
    g = torch.Generator().manual_seed(seed)
    w = {}
    for name, info in part.param_infos().items():
        t = torch.randn(info.shape, generator=g) * (0.2 if len(info.shape) > 1 else 0.5) + (1.0 if name == "norm" else 0.0)
        w[name] = (t if info.kind == "scalars" else t.to(torch.bfloat16)).to(DEV)
    part.load(w)
    return part


def _rows(part, lens, xs):
    """The layer's rows, before the output projection, of sequences that share one step, and the records' states behind it."""
    from rusty_llama_b200.cache import Cache

    from test_parts import ctx_for

    cache = Cache([(0, part.cache_need())], 64 * 16, len(lens), torch.bfloat16, DEV)
    slots = [cache.open_sequence() for _ in lens]
    step, tables = ctx_for(cache, slots, [0] * len(lens), lens)
    view = cache.view(0, tables)
    a, _ = part.forward_unprojected(torch.cat(xs), step, view)
    return list(a.split(lens)), [view[0].state[s].clone() for s in slots]


@pytest.mark.parametrize("dim, vdim", [(128, 128), (36, 72), (64, 20), (100, 4)])
def test_the_norm_taken_along_has_the_same_bits(dim, vdim):
    from rusty_llama_b200.kernels import ops

    lens, H, G = [130, 40], 2, 1
    q, k, v, beta, logd = inputs(lens, H, G, dim, vdim, 12, "usual")
    T, g = sum(lens), torch.Generator().manual_seed(3)
    rows = torch.randn(T, H * vdim + 4, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(vdim, generator=g).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    scratch = torch.empty(ops.delta_chunked_scratch_floats(T, 2, H, dim, vdim), device=DEV)

    def run(norm):
        return ops.delta_chunked(q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV), v.reshape(T, -1).to(DEV), beta.to(DEV), logd.to(DEV),
                                 torch.zeros(2, H, dim, vdim, device=DEV), i32([0, 1]), i32([0, 130, 170]), H, G, dim, vdim, 130, scratch, norm=norm)

    plain = run(None)
    for gate in (None, rows[:, 4:]):
        for act in (ops.GATE_NONE, ops.GATE_SIGMOID, ops.GATE_SILU):
            assert torch.equal(run((w, 1e-5, gate, act, 0.3, None)), ops.head_norm_gate(plain, H, vdim, w, 1e-5, gate, act, torch.bfloat16, out_scale=0.3))


def test_a_prompts_bits_do_not_depend_on_its_company():
    """A prompt alone, whose norm is in the last of the chunks' kernels, and beside sequences of few tokens, where it is a kernel of its own; and those
    few tokens, which keep to the kernels of single tokens and come out as they do beside another prompt."""
    part = _layer()
    g = torch.Generator().manual_seed(1)
    x = {n: torch.randn(n, 64, generator=g).to(torch.bfloat16).to(DEV) for n in (100, 5, 31, 200, 1)}
    (want,), (want_S,) = _rows(part, [100], [x[100]])
    (_, few), (_, few_S) = _rows(part, [200, 5], [x[200], x[5]])
    for lens in ([100, 5], [5, 100], [31, 100, 1, 5], [200, 5, 100], [100, 200]):
        got, got_S = _rows(part, lens, [x[n] for n in lens])
        assert torch.equal(got[lens.index(100)], want) and torch.equal(got_S[lens.index(100)], want_S), lens
        if 5 in lens:
            assert torch.equal(got[lens.index(5)], few) and torch.equal(got_S[lens.index(5)], few_S), lens


@pytest.mark.parametrize("lens, H, G, dim, vdim", [([200, 64, 1, 63], 4, 2, 128, 128), ([400], 2, 1, 100, 132), ([33, 300], 3, 3, 64, 20)])
def test_chunks_in_several_goes(lens, H, G, dim, vdim):
    """With room for one, two or three chunks of every sequence at a time: the same bits, results and states, and the same sequences left alone."""
    from rusty_llama_b200.errors import KernelError
    from rusty_llama_b200.kernels import ops

    q, k, v, beta, logd = inputs(lens, H, G, dim, vdim, 21, "usual")
    T, S = sum(lens), len(lens)
    starts = [sum(lens[:i]) for i in range(S + 1)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    first = torch.randn(S, H, dim, vdim, generator=torch.Generator().manual_seed(4)).to(DEV)
    gate, w = torch.randn(T, H * vdim, device=DEV).to(torch.bfloat16), torch.randn(vdim, device=DEV)
    full = ops.delta_chunked_scratch_floats(T, S, H, dim, vdim)
    a_chunk = full // (T // 64 + S + 1) * S

    def run(floats, norm, min_len):
        state, out = first.clone(), torch.zeros(T, H * vdim, dtype=torch.bfloat16, device=DEV)
        got = ops.delta_chunked(q.reshape(T, -1).to(DEV), k.reshape(T, -1).to(DEV), v.reshape(T, -1).to(DEV), beta.to(DEV), logd.to(DEV), state, i32(list(range(S))),
                                i32(starts), H, G, dim, vdim, max(lens), torch.full((floats,), float("nan"), device=DEV), min_len,
                                norm=(w, 1e-5, gate, ops.GATE_SILU, 1.0, out) if norm else None)
        return got, state

    for norm, min_len in ((False, 1), (vdim <= 128, 64)):
        want, want_S = run(full, norm, min_len)
        for chunks in (1, 2, 3):
            assert ops.delta_chunked_window(chunks * a_chunk, T, S, H, dim, vdim) == (chunks if chunks * a_chunk < full else 0)
            got, got_S = run(chunks * a_chunk, norm, min_len)
            for i, n in enumerate(lens):
                if n >= min_len:
                    assert torch.equal(got[starts[i] : starts[i + 1]], want[starts[i] : starts[i + 1]])
                elif norm:
                    assert not bool(got[starts[i] : starts[i + 1]].any())
            assert torch.equal(got_S, want_S)
    with pytest.raises(KernelError):
        run(a_chunk - 1, False, 1)


def test_a_step_with_little_memory_left_still_goes_by_chunks(monkeypatch):
    """Where the device has no room for the whole scratch, what the matrices take unsplit does, with the same bits; with less it is token by token."""
    import rusty_llama_b200.parts.gated_recurrent as module
    from rusty_llama_b200.kernels import ops

    part, before = _layer(), ops.delta_chunked
    x = torch.randn(700, 64, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(DEV)
    (want,), (want_S,) = _rows(part, [700], [x])
    full, less, called = ops.delta_chunked_scratch_floats(700, 1, 4, 32, 48), ops.delta_chunked_less_scratch_floats(700, 1, 4, 32, 48), []
    assert 3 * less < 2 * full
    monkeypatch.setattr(ops, "delta_chunked", lambda *a, **k: called.append(a[13].numel()) or before(*a, **k))
    for room, takes in ((full, full), (full - 1, less), (less, less), (less - 1, None)):
        called.clear()
        monkeypatch.setattr(module, "scratch_for_call", lambda n, dtype, device: torch.empty(n, dtype=dtype, device=device) if n <= room else None)
        (got,), (got_S,) = _rows(part, [700], [x])
        assert called == ([takes] if takes else [])
        if takes:
            assert torch.equal(got, want) and torch.equal(got_S, want_S)
        else:
            assert float((got_S - want_S).norm() / want_S.norm()) <= 1e-5

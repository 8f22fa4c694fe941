"""Prompt steps of the latent attention over keys and values expanded per head: the layer against 64 bits at sizes around the kernels'
padded ones, with keys of an earlier step, windows, ragged batches and without sink or gate; the rule that takes a step there; and the
prompt attention's roles giving up at a key size of 192, where there is one value stage."""

import math

import pytest
import torch

from test_parts import ctx_for
from test_waits import expect_give_up, with_memory_left

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def turn(x, f, first):
    """Pairs (i, i + n) of the leading 2 n numbers of x [T, ..., rot] turned by position * f."""
    n = len(f)
    angle = (torch.arange(x.shape[0], dtype=torch.float64) + first).view(-1, *([1] * (x.dim() - 1))) * f
    a, b = x[..., :n], x[..., n : 2 * n]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), x[..., 2 * n :]], dim=-1)


def make(H, dim, rot, vdim, rank, d, window=0, sink=True, gate=True, q_rank=0, dtype=torch.bfloat16):
    from rusty_llama_b200.parts import MIXERS, Runtime
    from rusty_llama_b200.spec import PartSpec

    pos = PartSpec("rotary", {"rotary_dim": rot, "theta": 500.0, "scaling": None, "interleaved": False}) if rot else PartSpec("none")
    part = MIXERS.build(PartSpec("latent_attention", {
        "hidden_size": d, "num_heads": H, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank, "scale": (dim + rot) ** -0.5, "eps": 1e-5,
        "sink": sink, "gate": gate, "window": window, "q_rank": q_rank, "position": pos}), Runtime.create(DEV, dtype))
    g = torch.Generator().manual_seed(dim + rot + vdim)
    w = {}
    for name, info in part.param_infos().items():
        t = torch.randn(info.shape, generator=g) / (math.sqrt(info.shape[-1]) if len(info.shape) > 1 else 2.0) + (1.0 if name.endswith("norm") else 0.0)
        w[name] = t.float() if info.kind == "scalars" else t.to(dtype)
    part.load({k: v.to(DEV) for k, v in w.items()})
    return part, {k: v.double() for k, v in w.items()}


def plain(w, x, H, dim, rot, vdim, rank, window, sink, gate, q_rank):
    f = 500.0 ** (-torch.arange(0, rot, 2, dtype=torch.float64) / max(rot, 1))
    rms = lambda t, g: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-5) * g  # noqa: E731
    q = (rms(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T if q_rank else x @ w["q"].T).view(-1, H, dim + rot)
    raw = x @ w["dkv"].T
    c, kr = rms(raw[:, :rank], w["dkv.norm"]), turn(raw[:, None, rank:], f, 0)
    q = torch.cat([q[..., :dim], turn(q[..., dim:], f, 0)], -1)
    k = torch.cat([(c @ w["uk"].T).view(-1, H, dim), kr.expand(-1, H, -1)], -1)
    v = (c @ w["uv"].T).view(-1, H, vdim)
    n = x.shape[0]
    s = torch.einsum("thd,shd->hts", q, k) * (dim + rot) ** -0.5
    back = torch.arange(n)[:, None] - torch.arange(n)[None]
    s = s.masked_fill((back < 0) | ((back >= window) if window else (back < 0)), float("-inf"))
    if sink:
        s = torch.cat([s, w["sink"][:, None, None].expand(H, n, 1)], -1)
    p = torch.softmax(s, -1)[..., :n]
    o = torch.einsum("hts,shd->thd", p, v).reshape(n, H * vdim)
    return (o * torch.sigmoid(x @ w["g"].T) if gate else o) @ w["o"].T


CASES = [
    # H, dim, rot, vdim, rank, options
    (4, 128, 64, 128, 512, {}),
    (4, 128, 64, 64, 512, {"window": 70}),
    (8, 64, 32, 64, 256, {}),
    (3, 40, 8, 24, 64, {"sink": False}),
    (2, 120, 16, 72, 128, {"gate": False}),
    (5, 64, 0, 128, 192, {"q_rank": 96}),
    (2, 16, 48, 8, 64, {"window": 33}),
]


@pytest.mark.parametrize("H, dim, rot, vdim, rank, options", CASES)
def test_prompts_in_two_steps(H, dim, rot, vdim, rank, options):
    from rusty_llama_b200.cache import Cache

    o = dict(dict(window=0, sink=True, gate=True, q_rank=0), **options)
    d = 96
    part, w = make(H, dim, rot, vdim, rank, d, **o)
    first, second = [130, 1, 64, 33], [65, 200, 1, 64]  # tokens of every sequence in the two steps
    g = torch.Generator().manual_seed(H)
    xs = [torch.randn(a + b, d, generator=g).to(torch.bfloat16) for a, b in zip(first, second)]
    cache = Cache([(0, part.cache_need())], 64 * 24, 4, torch.bfloat16, DEV)
    cache.kv_groups[0].k.normal_()  # (what pages held before must not matter)
    slots = [cache.open_sequence() for _ in first]
    want = [plain(w, x.double(), H, dim, rot, vdim, rank, **o) for x in xs]
    for lens, pos0 in ((first, [0] * 4), (second, first)):
        step, tables = ctx_for(cache, slots, pos0, lens)
        xn = torch.cat([x[p : p + n] for x, p, n in zip(xs, pos0, lens)]).to(DEV)
        assert part._expands(step, torch.empty(1, 8, device=DEV, dtype=torch.bfloat16), None) == (step.max_kv_len + 63) // 64 * 64
        got = part.forward(xn, step, cache.view(0, tables))
        got = (got.float().sum(0) if got.dim() == 3 else got.float()).cpu().double()
        ref = torch.cat([y[p : p + n] for y, p, n in zip(want, pos0, lens)])
        err = (got - ref).abs()
        assert float(err.max()) <= 1.5e-2 * float(ref.abs().max()) and float(err.mean()) <= 2.5e-3 * float(ref.abs().max())
        cache.commit(slots, lens)


def test_both_forms_of_a_step_agree():
    """The same prompts through the latents (the rule's limits set so that nothing expands) and expanded."""
    import rusty_llama_b200.parts.latent_attention as module
    from rusty_llama_b200.cache import Cache

    part, w = make(4, 128, 64, 128, 512, 128)
    g = torch.Generator().manual_seed(9)
    lens = [150, 77]
    x = torch.randn(sum(lens), 128, generator=g).to(torch.bfloat16).to(DEV)
    out = {}
    for least in (module._EXPAND_MIN_TOKENS, 10**9):
        cache = Cache([(0, part.cache_need())], 64 * 8, 2, torch.bfloat16, DEV)
        step, tables = ctx_for(cache, [cache.open_sequence() for _ in lens], [0, 0], lens)
        before, module._EXPAND_MIN_TOKENS = module._EXPAND_MIN_TOKENS, least
        try:
            y = part.forward(x, step, cache.view(0, tables))
        finally:
            module._EXPAND_MIN_TOKENS = before
        out[least] = (y.float().sum(0) if y.dim() == 3 else y.float()).double()
        out[least, "cache"] = cache.kv_groups[0].k.clone()
    a, b = (v for k, v in out.items() if not isinstance(k, tuple))
    assert float((a - b).norm() / b.norm()) < 1e-2
    c1, c2 = (v for k, v in out.items() if isinstance(k, tuple))
    assert torch.equal(c1, c2)


@pytest.mark.parametrize("code, text", [(11, "producer"), (12, "producer"), (14, "issuer"), (16, "issuer"), (17, "softmax")])
def test_a_role_gives_up_with_keys_of_192(code, text):
    from rusty_llama_b200.kernels import ops

    g = torch.Generator().manual_seed(code)
    H, n = 2, 300
    kv = torch.randn(320, H, 320, generator=g).to(torch.bfloat16).to(DEV)
    q = torch.randn(n, H * 192, generator=g).to(torch.bfloat16).to(DEV)
    start, pos0 = torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.tensor([0], dtype=torch.int32, device=DEV)
    run = lambda: ops.flash_expanded(q, kv, 320, start, pos0, n, 128, 0, 192 ** -0.5)  # noqa: E731
    before = run()
    expect_give_up(ops, code, "flash_prefill_tc: .*" + text, run)
    assert torch.equal(run(), before)
    ops.tc_status_check()


@pytest.mark.parametrize("H, dim, rot, vdim, rank", [(8, 64, 32, 64, 256), (4, 128, 64, 128, 512)])
def test_expanding_loses_nothing_against_64_bits(H, dim, rot, vdim, rank):
    """The gated sums of both forms of a step against 64 bits: rounding keys and values per head costs what rounding queries and sums in the
    latent space costs, and the probabilities must not cost more."""
    import rusty_llama_b200.parts.latent_attention as module
    from rusty_llama_b200.cache import Cache

    part, w = make(H, dim, rot, vdim, rank, 256)
    g = torch.Generator().manual_seed(17)
    lens = [41, 64, 222, 300]
    xs = [(2 * torch.randn(n, 256, generator=g)).to(torch.bfloat16) for n in lens]
    want = torch.cat([plain(dict(w, o=torch.eye(H * vdim, dtype=torch.float64)), x.double(), H, dim, rot, vdim, rank, 0, True, True, 0) for x in xs])
    off = []
    for least in (module._EXPAND_MIN_TOKENS, 10**9):
        cache = Cache([(0, part.cache_need())], 64 * 12, 4, torch.bfloat16, DEV)
        step, tables = ctx_for(cache, [cache.open_sequence() for _ in lens], [0] * 4, lens)
        before, module._EXPAND_MIN_TOKENS = module._EXPAND_MIN_TOKENS, least
        try:
            a, _ = part.forward_unprojected(torch.cat(xs).to(DEV), step, cache.view(0, tables))
        finally:
            module._EXPAND_MIN_TOKENS = before
        off.append(float((a.double().cpu() - want).norm() / want.norm()))
    assert off[0] <= off[1], off


def test_a_step_without_room_for_the_rows_works_on_the_latents():
    import rusty_llama_b200.parts.latent_attention as module
    from rusty_llama_b200.cache import Cache

    part, w = make(16, 128, 64, 128, 512, 96)
    held, n = 8000, 256
    cache = Cache([(0, part.cache_need())], 64 * 130, 1, torch.bfloat16, DEV)
    cache.kv_groups[0].k.normal_(generator=torch.Generator(device=DEV).manual_seed(1))
    slot = cache.open_sequence()
    cache.reserve([slot], [held])
    cache.commit([slot], [held])
    step, tables = ctx_for(cache, [slot], [held], [n])
    x = torch.randn(n, 96, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(DEV)
    run = lambda: part.forward(x, step, cache.view(0, tables))  # noqa: E731
    before, module._EXPAND_MIN_TOKENS = module._EXPAND_MIN_TOKENS, 10**9
    try:
        want = run()
    finally:
        module._EXPAND_MIN_TOKENS = before
    assert part._expands(step, torch.empty(1, 8, device=DEV, dtype=torch.bfloat16), None)
    scratch = 2 * (held + n) * (16 * 320 + 512)
    assert torch.equal(with_memory_left(scratch - (8 << 20), run), want)


@pytest.mark.parametrize("vdim", [8, 64, 72, 128])
def test_output_gates_of_every_size(vdim):
    """The gate beside whole row blocks, short ones and one of a single row: logistic functions of large gates, of infinite ones and of what is no
    number, which stays in its place.  Against the same without a gate, whose result is rounded too: 2^-8 of it at most, twice."""
    from rusty_llama_b200.kernels import ops

    lens, H, rows = [128, 33, 129, 1], 2, 192
    T, dim = sum(lens), 64
    g = torch.Generator().manual_seed(vdim)
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kv = torch.randn(rows * len(lens), H, dim + vdim, generator=g).to(torch.bfloat16).to(DEV)
    q = torch.randn(T, H * dim, generator=g).to(torch.bfloat16).to(DEV)
    gate = torch.randn(T, H * vdim + 8, generator=g) * 4
    for value in (float("inf"), float("-inf"), float("nan"), 100.0, -100.0, -80.0):
        gate.view(-1)[torch.randperm(gate.numel(), generator=g)[:40]] = value
    gate[starts[2] - 1, 0], gate[T - 1, vdim - 1] = float("nan"), float("-inf")
    gate = gate.to(torch.bfloat16).to(DEV)[:, : H * vdim]
    args = (q, kv, rows, i32(starts), i32([0] * len(lens)), max(lens), vdim, 0, dim ** -0.5)
    plain, got = ops.flash_expanded(*args).double(), ops.flash_expanded(*args, gate=gate).double()
    want = plain * torch.sigmoid(gate.double())
    assert torch.equal(got.isnan(), want.isnan())
    assert bool(((got - want).abs() <= want.abs() * (2.0 ** -7 * 1.01) + 1e-38)[~want.isnan()].all())

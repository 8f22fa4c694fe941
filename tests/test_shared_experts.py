"""Matrices that take every token beside a routed feed-forward's experts: the plan's rows and tiles, the sum, the whole part against
the plain sum in 32-bit; and the choice from partial sums of the logits."""

import pytest
import torch

from rusty_llama_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T, top, E, always, rows", [(1, 1, 1, 1, 32), (1, 2, 4, 2, 32), (33, 2, 5, 1, 32), (96, 4, 32, 1, 32), (300, 3, 7, 2, 128), (2048, 6, 64, 2, 256), (257, 6, 64, 3, 128), (601, 7, 40, 1, 128), (64, 2, 600, 1, 32)])
def test_plan(T, top, E, always, rows):
    g = torch.Generator().manual_seed(T + E)
    ids = torch.stack([torch.randperm(max(E, top), generator=g)[:top] for _ in range(T)]).to(torch.int32)
    if E > 4:
        ids[0, 0] = E + 1  # names no expert
    order, place, tiles, most = ops.moe_plan(ids.to(DEV), E, rows, always)
    order, place, tiles = order.cpu(), place.cpu(), tiles.cpu()
    n, count = T * top, int(tiles[0])
    assert count <= most
    seen = torch.zeros(n + always * T, dtype=torch.int32)
    owner = torch.full((n + always * T,), -1)
    at = []
    for i, (e, r0, k) in enumerate(tiles[1 : 1 + 3 * count].view(-1, 3).tolist()):
        assert 0 < k <= rows and 0 <= e < E + always
        seen[r0 : r0 + k] += 1
        owner[r0 : r0 + k] = e
        at += [i] if e >= E else []
    flat = ids.flatten()
    held = int((flat < E).sum())
    assert bool((seen[:held] == 1).all()) and bool((seen[held:n] == 0).all()) and bool((seen[n:] == 1).all())
    for p in range(n):
        r = int(place[p])
        assert r == -1 if flat[p] >= E else (int(order[r]) == p and owner[r] == flat[p])
    for j in range(always):
        assert torch.equal(order[n + j * T : n + (j + 1) * T], torch.arange(T, dtype=torch.int32) * top) and bool((owner[n + j * T : n + (j + 1) * T] == E + j).all())
    # the tiles of all tokens stand evenly between the others
    steps = [b - a for a, b in zip(at, at[1:])]
    assert not steps or max(steps) - min(steps) <= 1


@pytest.mark.parametrize("E, top", [(1, 1), (31, 3), (32, 32), (33, 2), (64, 6), (65, 33), (128, 8), (200, 4), (256, 40), (512, 9), (600, 5), (1000, 7), (1536, 2)])
@pytest.mark.parametrize("parts, gated, logistic, renorm", [(1, False, False, True), (3, True, True, False), (8, True, False, True)])
def test_choice_from_partial_sums(E, top, parts, gated, logistic, renorm):
    """Scores are one exponential and one division off the oracle's: 1e-5 (the sum over E experts rounds 11 times at most); choices differ
    nowhere, scores being apart by more than that or equal (then the lower index is chosen)."""
    T = 37
    g = torch.Generator().manual_seed(E + parts)
    rows = E + int(gated)
    z = torch.randint(-40, 41, (parts, T, rows), generator=g).float() / 16 / parts  # (many ties)
    bias = torch.randint(-2, 3, (E,), generator=g).float() / 4
    ids, weights, gate = ops.moe_choose(z.to(DEV) if parts > 1 else z[0].to(DEV), bias.to(DEV), E, top, renormalize=renorm, logistic=logistic, renorm_eps=0.25, weight_scale=1.5)
    whole = z[0].clone()
    for p in range(1, parts):
        whole += z[p]
    x = whole[:, :E].double()
    score = torch.sigmoid(x) if logistic else torch.softmax(x, dim=1)
    key = score.float() + bias  # (the oracle rounds where the kernel does; equal logits have equal scores on both sides)
    want = torch.sort(key, dim=1, descending=True, stable=True)[1][:, :top]
    got = ids.cpu().long()
    picked, best = key.gather(1, got), key.gather(1, want)
    assert float((picked - best).abs().max()) <= 1e-6  # (two keys closer than the scores' own roundings may change places)
    assert all(len(set(r.tolist())) == top for r in got)
    s = score.gather(1, got)
    w = (s / (s.sum(1, keepdim=True) + 0.25) if renorm else s) * 1.5
    assert float((weights.cpu().double() - w).abs().max()) <= 1e-5
    if gated:
        assert float((gate.cpu().double() - torch.sigmoid(whole[:, E].double())).abs().max()) <= 1e-6


def test_scores_that_are_no_numbers_choose_each_expert_once():
    z = torch.zeros(3, 40)
    z[0] = float("nan")
    z[1, 7] = float("nan")
    z[2, 5] = float("inf")
    ids, _, _ = ops.moe_choose(z.to(DEV), None, 40, 33)
    for row in ids.cpu().tolist():
        assert len(set(row)) == 33 and all(0 <= e < 40 for e in row)


@pytest.mark.parametrize("T", [1, 5, 8, 9, 40, 200])
@pytest.mark.parametrize("shared_ff, gated", [(64, False), (192, True), (96, True)])
def test_part(T, shared_ff, gated):
    """All of a shared expert's forms (of the experts' size, of a multiple of it, of another size) against the plain sum in 32 bits: the
    hidden rows are rounded to bfloat16 (2^-9 of each, at random), and so is a shared expert's result."""
    from rusty_llama_b200.parts import FEED_FORWARDS, Runtime
    from rusty_llama_b200.spec import PartSpec

    d, E, top, ff = 128, 6, 2, 64
    part = FEED_FORWARDS.build(PartSpec("routed_experts", {"hidden_size": d, "n_experts": E, "top": top, "expert_ff": ff, "bias": False, "renormalize": True,
                                                           "shared_ff": shared_ff, "shared_gate": gated}), Runtime.create(DEV, torch.bfloat16))
    g = torch.Generator().manual_seed(shared_ff)
    w = {}
    for name, info in part.param_infos().items():
        t = (torch.randn(info.shape, generator=g) * info.shape[-1] ** -0.5).to(torch.bfloat16)
        w[name] = (t.float() if info.kind == "scalars" else t).to(DEV)
    part.load(w)
    assert part.always == (shared_ff // ff if shared_ff % ff == 0 else 0) and part._joins(T) == (8 <= T <= 192)
    x = torch.randn(T, d, generator=g).to(torch.bfloat16).to(DEV)
    got = part.forward(x, None).float()
    f = {k: v.float() for k, v in w.items()}
    xf = x.float()
    mlp = lambda y, p: (torch.nn.functional.silu(y @ f[p + "gate"].T) * (y @ f[p + "up"].T)) @ f[p + "down"].T  # noqa: E731
    score, chosen = torch.softmax(xf @ f["router"].T, dim=1).topk(top, dim=1)
    score = score / score.sum(1, keepdim=True)
    want = mlp(xf, "shared.") * (torch.sigmoid(xf @ f["shared.sg"].T) if gated else 1.0)
    for e in range(E):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            want.index_add_(0, rows, mlp(xf[rows], f"e{e}.") * score[rows, place, None])
    assert float((got - want).norm() / want.norm()) <= 8e-3


@pytest.mark.parametrize("d, ff", [(128, 64), (136, 64), (64, 200), (328, 72)])  # (whole tiles of features and slices of k, and parts of them)
@pytest.mark.parametrize("pieces, gated", [(1, False), (3, True)])
def test_a_shared_experts_way_does_not_show(d, ff, pieces, gated, monkeypatch):
    """The same tokens with the shared expert's rows in the experts' products and in products of their own.  Both round its result to
    bfloat16; their 32-bit sums differ by some 2^-22, which puts one number in 2^13 on the other side of a rounding, 2^-8 off: 5e-5 in
    all, twice that allowed.  (Unrounded on one of the ways it is 1e-3.)"""
    from rusty_llama_b200.parts import FEED_FORWARDS, Runtime
    from rusty_llama_b200.spec import PartSpec

    part = FEED_FORWARDS.build(PartSpec("routed_experts", {"hidden_size": d, "n_experts": 6, "top": 2, "expert_ff": ff, "bias": False, "renormalize": True,
                                                           "shared_ff": pieces * ff, "shared_gate": gated}), Runtime.create(DEV, torch.bfloat16))
    g = torch.Generator().manual_seed(pieces + d)
    w = {}
    for name, info in part.param_infos().items():
        t = (torch.randn(info.shape, generator=g) * info.shape[-1] ** -0.5).to(torch.bfloat16)
        w[name] = (t.float() if info.kind == "scalars" else t).to(DEV)
    part.load(w)
    x = torch.randn(150, d, generator=g).to(torch.bfloat16).to(DEV)
    assert part.always and part._joins(150)
    joined = part.forward(x, None).double()
    monkeypatch.setattr(part, "_joins", lambda T: False)
    apart = part.forward(x, None).double()
    assert float((joined - apart).norm() / apart.norm()) <= 1e-4


@pytest.mark.parametrize("d", [6, 8])  # (rows of whole fours have a kernel of their own)
@pytest.mark.parametrize("always, gated", [(1, True), (3, False), (9, True)])
def test_sum_of_the_matrices_that_take_every_token(d, always, gated):
    T, top = 5, 2
    g = torch.Generator().manual_seed(d + always)
    y = torch.randn(T * (top + always), d, generator=g)
    place = torch.randperm(T * top, generator=g).to(torch.int32)
    weights, gate = torch.rand(T, top, generator=g), torch.rand(T, generator=g)
    got = ops.moe_combine(y.to(DEV), place.to(DEV), weights.to(DEV), None, gate.to(DEV) if gated else None, always=always).cpu()
    own = torch.zeros(T, d)
    for j in range(always):
        own += y[T * (top + j) : T * (top + j + 1)]
    want = (weights.double()[:, :, None] * y.double()[place.long()].view(T, top, d)).sum(1) + own.to(torch.bfloat16).double() * (gate.double()[:, None] if gated else 1.0)
    assert float((got.double() - want).abs().max()) <= 4 * 2.0**-24 * 8  # (four roundings of numbers below eight)

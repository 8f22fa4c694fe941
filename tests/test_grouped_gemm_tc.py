"""The grouped products on tcgen05: row tiles at the edges of their heights (none, one row, a multiple of 16 and one more, several tiles
of an expert), features and k that leave remainders, each way out; products per head at the same edges; and the give-up paths."""

import pytest
import torch

from test_waits import expect_give_up

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from rusty_llama_b200.kernels import ops

    return ops


def ids_for(counts, top):
    """Choices [T, top] in which expert e is named counts[e] times, spread over the tokens."""
    named = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)], dtype=torch.int32)
    assert named.numel() % top == 0
    return named.view(top, -1).t().contiguous()


def close(got, want, mag, K, out_rounds):
    """32-bit sums of K exact products (each rounding at most 2^-24 of the sum of magnitudes; the tensor core may truncate: twice that),
    then a rounding of the result to its type."""
    tol = K * 2.0 ** -23 * mag + (2.0 ** -8 if out_rounds else 0.0) * want.abs() + 1e-30
    assert bool(((got.double().cpu() - want).abs() <= tol).all()), float(((got.double().cpu() - want).abs() / tol).max())


# counts of rows per expert: tile heights of 32, 128 and 256 and what is around them
COUNTS = {
    32: [0, 1, 15, 16, 17, 31, 32, 33, 0, 64, 70, 3],
    128: [127, 0, 128, 129, 16, 1, 257, 100],
    256: [255, 256, 257, 0, 300, 512, 513, 1, 240, 176],
}


@pytest.mark.parametrize("N, K", [(128, 64), (200, 72), (64, 8), (1408, 264), (40, 520)])
@pytest.mark.parametrize("tile_rows", [32, 128, 256])
def test_experts_products(ops, tile_rows, N, K):
    g = torch.Generator().manual_seed(tile_rows + N + K)
    counts = list(COUNTS[tile_rows])
    top = 2
    if sum(counts) % top:
        counts[-1] += 1
    E, ids = len(counts), ids_for(counts, top)
    T = ids.shape[0]
    order, place, tiles, mt = ops.moe_plan(ids.to(DEV), E, tile_rows)
    o, tl = order.cpu().long(), tiles.cpu().tolist()
    covered = torch.zeros(T * top, dtype=torch.int64)
    for i in range(tl[0]):
        e, r0, n = tl[1 + 3 * i : 4 + 3 * i]
        assert 0 < n <= tile_rows and bool((ids.reshape(-1)[o[r0 : r0 + n]] == e).all())
        covered[r0 : r0 + n] += 1
    assert bool((covered == 1).all()) and tl[0] == sum((c + tile_rows - 1) // tile_rows for c in counts)
    rand = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)  # noqa: E731
    x, w, w2 = rand(T, K + 8), rand(E, N, K), rand(E, N, K)
    xd = x.to(DEV)[:, :K]  # rows further apart than they are long
    rows, expert = x[:, :K].double()[o // top], ids.reshape(-1)[o].long()
    prod = lambda m: torch.stack([rows[i] @ m[expert[i]].double().T for i in range(T * top)])  # noqa: E731
    mag = lambda m: torch.stack([rows[i].abs() @ m[expert[i]].double().abs().T for i in range(T * top)])  # noqa: E731
    a, b, ma, mb = prod(w), prod(w2), mag(w), mag(w2)
    run = lambda **kw: ops.moe_gemm(xd, w.to(DEV), tiles, mt, T * top, order=order, gather_div=top, tile_rows=tile_rows, **kw)  # noqa: E731
    close(run(out_dtype=torch.float32), a, ma, K, False)
    close(run(act="relu2"), a.clamp(min=0) ** 2, 2 * a.abs() * ma, K, True)
    close(run(w2=w2.to(DEV)), a * torch.sigmoid(a) * b, 1.1 * ma * b.abs() + a.abs() * mb, K, True)
    # the plan's rows as they are (the second product of a feed-forward)
    h = rand(T * top, K)
    want = torch.stack([h[i].double() @ w[expert[i]].double().T for i in range(T * top)])
    got = ops.moe_gemm(h.to(DEV), w.to(DEV), tiles, mt, T * top, out_dtype=torch.float32, tile_rows=tile_rows)
    close(got, want, torch.stack([h[i].double().abs() @ w[expert[i]].double().abs().T for i in range(T * top)]), K, False)
    ops.tc_status_check()


def test_more_tiles_than_are_listed_in_shared_memory(ops):
    g = torch.Generator().manual_seed(3)
    E, K, N = 700, 64, 128
    ids = torch.arange(E, dtype=torch.int32)[:, None].to(DEV)
    x, w = torch.randn(E, K, generator=g).to(torch.bfloat16), torch.randn(E, N, K, generator=g).to(torch.bfloat16)
    order, place, tiles, mt = ops.moe_plan(ids, E, 32)
    got = ops.moe_gemm(x.to(DEV), w.to(DEV), tiles, mt, E, order=order, out_dtype=torch.float32, tile_rows=32)
    close(got, torch.einsum("ek,enk->en", x.double(), w.double()), torch.einsum("ek,enk->en", x.double().abs(), w.double().abs()), K, False)


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("M, H, N, K", [(33, 3, 128, 64), (255, 2, 72, 40), (256, 1, 512, 128), (257, 5, 64, 136), (600, 2, 130, 512)])
def test_products_per_head(ops, M, H, N, K, gated):
    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn(M, H * (K + 8), generator=g).to(torch.bfloat16), torch.randn(H, N, K, generator=g).to(torch.bfloat16)
    gate = torch.randn(M, H * N, generator=g).to(torch.bfloat16) if gated else None
    out = torch.full((M, H * (N + 2)), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.head_linear(x.to(DEV), K + 8, w.to(DEV), out, N + 2, gate=None if gate is None else gate.to(DEV), gate_head_stride=N)
    xs = x.view(M, H, K + 8)[:, :, :K].double()
    want, mag = torch.einsum("mhk,hnk->mhn", xs, w.double()), torch.einsum("mhk,hnk->mhn", xs.abs(), w.double().abs())
    if gated:
        s = torch.sigmoid(gate.view(M, H, N).double())
        want, mag = want * s, mag * s
    got = out.view(M, H, N + 2)
    close(got[:, :, :N], want, mag, K, True)
    assert bool((got[:, :, N:] == 7.0).all())


@pytest.mark.parametrize("code, text", [(61, "the copying lane"), (62, "the tensor-core issuer"), (63, "a result warp"), (65, "a gathering warp")])
def test_a_role_gives_up_and_the_next_launch_is_right(ops, code, text):
    g = torch.Generator().manual_seed(code)
    E, K, N, rows = 5, 1024, 1500, 300
    ids = ids_for([rows] * E, 2).to(DEV)
    order, place, tiles, mt = ops.moe_plan(ids, E, 128)
    x, w = torch.randn(E * rows // 2, K, generator=g).to(torch.bfloat16).to(DEV), torch.randn(E, N, K, generator=g).to(torch.bfloat16).to(DEV)
    run = lambda: ops.moe_gemm(x, w, tiles, mt, E * rows, order=order, gather_div=2, out_dtype=torch.float32, tile_rows=128)  # noqa: E731
    before = run()
    expect_give_up(ops, code, "grouped_gemm_tc: " + text, run)
    assert torch.equal(run(), before)
    ops.tc_status_check()


@pytest.mark.parametrize("tile_rows", [32, 128, 256])
def test_a_gate_far_below_zero(ops, tile_rows):
    """silu and the form with limits where 1 + exp(-gate) is above 2^126: the quotient is small and not zero (an approximate division
    gives zero there), within the result's rounding to bfloat16 (8 significant bits: 2^-8) and a few of 32 bits before it."""
    gates = torch.tensor([-1.0, -20.0, -60.0, -80.0, -86.0, -87.5, -88.0, -88.5, 0.0, 3.0, 40.0, 88.0] + [-87.5] * 52)
    N, K, T = gates.numel(), 8, 3
    x, w, w2 = torch.zeros(T, K), torch.zeros(2, N, K), torch.zeros(2, N, K)
    x[:, 0] = 1.0
    w[:, :, 0], w2[:, :, 0] = gates, 1.0
    bf = lambda t: t.to(torch.bfloat16).to(DEV)  # noqa: E731
    ids = torch.tensor([[0], [1], [0]], dtype=torch.int32, device=DEV)
    order, place, tiles, mt = ops.moe_plan(ids, 2, tile_rows)
    g = gates.double()
    for act, want in ((None, g / (1 + torch.exp(-g))), ((1.0, 100.0), g / (1 + torch.exp(-g)) * 2.0)):
        got = ops.moe_gemm(bf(x), bf(w), tiles, mt, T, order=order, w2=bf(w2), tile_rows=tile_rows, act=act).double().cpu()
        assert bool(((got - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs()).all()), (act, (got[0] / want).tolist()[:12])

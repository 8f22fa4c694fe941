"""The 32-bit products and the 32-bit attention: each launch form (few rows or many, tiles of every size, rows that cannot be moved
16 bytes at a time; heads of a kv head together or alone) against 64 bits, and against the other forms bit for bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from rusty_llama_b200.kernels import ops

    return ops


def product_bound(x, w):
    """A sum of K products in chunks of 128: each result is off by at most (128 + K / 128 + 1) roundings of what is added up so far,
    which is never more than sum |x w|."""
    K = x.shape[1]
    return (130 + K / 128) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("K", [4, 124, 128, 132, 516, 2048, 5632])
@pytest.mark.parametrize("N", [1, 37, 296, 700])
@pytest.mark.parametrize("M", [1, 2, 3, 7, 16, 17, 70])
def test_product_in_every_form(ops, M, N, K):
    g = torch.Generator().manual_seed(M * 7919 + N * 31 + K)
    x, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    xd, wd = x.to(DEV), w.to(DEV)
    out = ops.gemm_f32(xd, wd)
    assert bool(((out.cpu().double() - x.double() @ w.double().T).abs() <= product_bound(x, w)).all())
    # rows that start off a 16-byte boundary take the tile kernel's scalar loads: the same bits
    wide = torch.zeros(M, K + 1, device=DEV)
    wide[:, 1:] = xd
    assert torch.equal(ops.gemm_f32(wide[:, 1:], wd), out)
    # among many rows (larger tiles), and alone
    many = torch.cat([xd, torch.randn(4000, K, generator=g).to(DEV)])
    for rows in (400, 1000, 4000):
        assert torch.equal(ops.gemm_f32(many[: M + rows], wd)[:M], out)
    assert torch.equal(ops.gemm_f32(xd[M - 1 :], wd)[0], out[M - 1])


def test_product_of_a_very_long_k(ops):
    """The longest rows of the few-row kernel (338 chunks of 128 and one row of a block's shared memory) and ones too long for it, which go to
    the tile kernel however few they are: the same bits as among many rows."""
    g = torch.Generator().manual_seed(5)
    for K in (20000, 41856, 41860, 43264, 43268, 70000):
        x, w = torch.randn(12, K, generator=g), torch.randn(9, K, generator=g)
        xd, wd = x.to(DEV), w.to(DEV)
        many = ops.gemm_f32(xd, wd)
        assert bool(((many.cpu().double() - x.double() @ w.double().T).abs() <= product_bound(x, w)).all())
        for rows in (1, 3, 8):
            assert torch.equal(ops.gemm_f32(xd[:rows], wd), many[:rows])


@pytest.mark.parametrize("N, K", [(2560, 2048), (2553, 1924), (11264, 2048), (40001, 2048), (2048, 5632), (2047, 14336), (16384, 3072), (9001, 3712),
                                  (1500, 41856), (1000, 43264)])
@pytest.mark.parametrize("M", [1, 2, 4, 5, 8])
def test_few_rows_of_large_matrices(ops, M, N, K):
    """Three blocks an SM, two and one, one pass and many, one wave of blocks and several, the most sums a block holds, the last block's fewer
    features: the same bits as among many rows."""
    g = torch.Generator(device=DEV).manual_seed(M * 7919 + N + K)
    x, w = torch.randn(40, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    assert torch.equal(ops.gemm_f32(x[:M], w), ops.gemm_f32(x, w)[:M])


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("H, K, hd", [(8, 1, 64), (6, 2, 40), (16, 2, 128), (5, 5, 30), (6, 1, 256), (12, 4, 18)])
def test_attention_of_few_and_of_many_tokens(ops, H, K, hd, window):
    g = torch.Generator().manual_seed(H * 100 + hd + window)
    L = 600
    pages = (L + 63) // 64
    k, v = torch.randn(L, K, hd, generator=g), torch.randn(L, K, hd, generator=g)
    order = torch.randperm(pages, generator=g)
    k_pages, v_pages = torch.zeros(pages, K, 64, hd), torch.zeros(pages, K, 64, hd)
    for i in range(L):
        k_pages[order[i // 64], :, i % 64], v_pages[order[i // 64], :, i % 64] = k[i], v[i]
    table = order.to(torch.int32)[None].to(DEV)
    pos = torch.cat([torch.arange(0, 100), torch.arange(250, 330), torch.arange(L - 120, L)]).to(torch.int32)
    q = torch.randn(len(pos), H * hd, generator=g)
    seq = torch.zeros(len(pos), dtype=torch.int32)
    args = (k_pages.to(DEV), v_pages.to(DEV), table)
    many = ops.attn_generic(q.to(DEV), *args, seq.to(DEV), pos.to(DEV), H, K, hd, window=window)
    n = len(pos)
    scores = torch.einsum("thd,khd->htk", q.view(n, H, hd).double(), k.repeat_interleave(H // K, 1).double()) / hd ** 0.5
    back = pos[:, None] - torch.arange(L)[None]
    scores = scores.masked_fill((back < 0) | ((back >= window) if window else (back < 0)), float("-inf"))
    ref = torch.einsum("htk,khd->thd", torch.softmax(scores, -1), v.repeat_interleave(H // K, 1).double()).reshape(n, H * hd)
    # a weight is off by the rounding of its score (hd terms of at most 6 in all) and of exp (2 ulp) and of the sums (32 terms, then groups, then
    # warps): relative 2^-24 times (6 hd + 70), and no result exceeds the largest value
    bound = 2.0 ** -24 * (hd * 6.0 + 70) * float(v.abs().max())
    assert float((many.cpu().double() - ref).abs().max()) <= bound
    for i in (0, 1, 31, 32, 99, 100, n - 1):  # one token: other heads per block, the same bits
        one = ops.attn_generic(q[i : i + 1].to(DEV), *args, seq[i : i + 1].to(DEV), pos[i : i + 1].to(DEV), H, K, hd, window=window)
        assert torch.equal(one[0], many[i])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_over_pages_that_start_anywhere(ops, dtype):
    """Pages in the middle of a larger buffer, off the boundary that four numbers at a time need: the same bits."""
    H, K, hd, L = 8, 2, 64, 150
    g = torch.Generator().manual_seed(3)
    pages = torch.randn(3, K, 64, hd, generator=g).to(dtype).to(DEV)
    q = torch.randn(L, H * hd, generator=g).to(dtype).to(DEV)
    table, seq = torch.arange(3, dtype=torch.int32, device=DEV)[None], torch.zeros(L, dtype=torch.int32, device=DEV)
    pos = torch.arange(L, dtype=torch.int32, device=DEV)
    want = ops.attn_generic(q, pages, pages, table, seq, pos, H, K, hd)
    for off in (1, 2, 3):
        buffer = torch.zeros(pages.numel() + off, dtype=dtype, device=DEV)
        moved = buffer[off:].view(pages.shape)
        moved.copy_(pages)
        assert torch.equal(ops.attn_generic(q, moved, moved, table, seq, pos, H, K, hd), want)


@pytest.mark.parametrize("hd, H, K", [(64, 4, 1), (60, 2, 2), (33, 3, 3), (4, 6, 2)])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_head_alone_asks_ahead(ops, hd, H, K, window, dtype):
    """Single tokens (reads ahead, no more blocks than the SMs hold) at the borders of the groups of 32 keys and of the warps' rounds: the same
    bits as among 400 tokens (no reads ahead)."""
    g = torch.Generator().manual_seed(hd + window)
    n, page = 560, 64
    pages = -(-n // page)
    k, v = (torch.randn(pages, K, page, hd, generator=g).to(DEV, dtype) for _ in range(2))
    table = torch.randperm(pages, generator=g).to(torch.int32).view(1, -1).to(DEV)
    at = [0, 1, 30, 31, 32, 33, 63, 64, 255, 256, 257, 288, 511, 512, 559]
    q = torch.randn(400, H * hd, generator=g).to(DEV, dtype)
    pos = torch.tensor((at * 27)[:400], dtype=torch.int32, device=DEV)
    run = lambda lo, hi: ops.attn_generic(  # noqa: E731
        q[lo:hi], k, v, table, torch.zeros(hi - lo, dtype=torch.int32, device=DEV), pos[lo:hi], H, K, hd, window=window, scale=hd ** -0.5)
    many = run(0, 400)
    for i in range(len(at)):
        assert torch.equal(run(i, i + 1)[0], many[i]), at[i]

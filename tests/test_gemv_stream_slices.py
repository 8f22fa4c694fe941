"""Products with few rows whose k comes in several slices: at a slice's end some warps load the next slice's activations while others
still read the ring's stages, and a stage may be copied over only once everyone has read it."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M, K, N", [(8, 14336, 2048), (8, 14336, 4096), (16, 13824, 2048), (3, 10240, 1000)])
def test_every_call_has_the_same_bits(M, K, N):
    from rusty_llama_b200.kernels import ops

    g = torch.Generator().manual_seed(K + N)
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16), (0.01 * torch.randn(N, K, generator=g)).to(torch.bfloat16)
    xd, wd = x.to(DEV), w.to(DEV)
    first = ops.gemv_stream(xd, wd, torch.float32, k_splits=2)
    differ = sum((ops.gemv_stream(xd, wd, torch.float32, k_splits=2) != first).any().int() for _ in range(300))
    assert int(differ) == 0
    # 32-bit sums of exact products: at most K roundings, each of at most 2^-24 of the sum of magnitudes
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((first.double().sum(0).cpu() - x.double() @ w.double().T).abs() <= bound).all())


@pytest.mark.parametrize("M, K, N", [(8, 4096, 8192), (1, 2048, 4096), (7, 5120, 5120), (16, 4096, 6144)])
def test_one_slice_every_call_has_the_same_bits(M, K, N):
    from rusty_llama_b200.kernels import ops

    g = torch.Generator().manual_seed(K + N + M)
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV), (0.02 * torch.randn(N, K, generator=g)).to(torch.bfloat16).to(DEV)
    for kw in ({"out_dtype": torch.float32}, {"swiglu": True}):
        first = ops.gemv_stream(x, w, **kw)
        differ = sum((ops.gemv_stream(x, w, **kw) != first).any().int() for _ in range(200))
        assert int(differ) == 0


@pytest.mark.parametrize("M, K, N", [(8, 4096, 8192), (8, 5120, 5120), (2, 2048, 7000)])
def test_into_the_stream_every_call_has_the_same_bits(M, K, N):
    """The folded form, whose storing warps read the stream and the next norm's weights beside the ring (more than four items a block
    at 7000 features and above: those beyond are read at the item's end)."""
    from rusty_llama_b200.kernels import ops

    g = torch.Generator().manual_seed(K + N)
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16), (0.02 * torch.randn(N, K, generator=g)).to(torch.bfloat16)
    before, nw = torch.randn(M, N, generator=g), torch.randn(N, generator=g)
    xd, wd, bd, nd = x.to(DEV), w.to(DEV), before.to(DEV), nw.to(DEV)

    def call():
        stream = bd.clone()
        xw, shares, blocks = ops.gemv_stream_into_stream(xd, wd, stream, nd)
        return stream, xw, shares[: blocks * 8].clone()

    first = call()
    differ = 0
    for _ in range(200):
        differ = differ + sum((a != b).any().int() for a, b in zip(call(), first))
    assert int(differ) == 0
    want = before.double() + x.double() @ w.double().T
    # at most K + 1 roundings of 2^-24 of the sum of magnitudes
    bound = (K + 1) * 2.0 ** -24 * (before.double().abs() + x.double().abs() @ w.double().abs().T)
    assert bool(((first[0].double().cpu() - want).abs() <= bound).all())

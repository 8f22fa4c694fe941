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

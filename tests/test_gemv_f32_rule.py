"""Which rows of x a block of the 32-bit streaming product takes: as many as there are, up to four, wherever the weights are what its time
goes for, since every group of rows reads them all again; and which products it takes at all."""

import shutil

import pytest

from rusty_llama_b200.kernels import host

SMS = 148


@pytest.fixture(scope="module")
def streams():
    if not shutil.which("nvcc"):
        pytest.skip("no CUDA compiler")
    return host.library("gemm_f32").rl_gemm_f32_streams


def before(M, N, K):
    """The rows a block of the rule that kept features and shared memory apart: 512 sums a row of x at most."""
    chunks = -(-K // 128)
    R, mb = min(-(-N // (2 * SMS)), 512 // chunks), 1 if M == 1 else 2 if M == 2 else 4
    need = lambda: 3 * 128 * 36 * 4 + mb * chunks * (132 + R) * 4  # noqa: E731
    while mb > 1 and need() > 112 * 1024:
        mb //= 2
    return mb if R > 0 and need() <= 224 * 1024 else 0


@pytest.mark.parametrize("N, K", [(40001, 2048), (128256, 2048), (32000, 2560), (16384, 3072), (128256, 3072), (11264, 2048), (2048, 5632)])
def test_the_weights_are_read_as_seldom_as_they_can_be(streams, N, K):
    for M in (1, 2, 3, 4, 5, 8):
        assert streams(M, N, K, SMS) >= before(M, N, K)
    if K <= 3072:
        assert streams(3, N, K, SMS) == streams(8, N, K, SMS) == 4


def test_what_was_streamed_is_streamed(streams):
    for K in list(range(4, 45000, 1988)) + [41856, 43264, 43268, 70000]:
        for N in (1, 9, 296, 297, 1000, 4096, 40001, 200000):
            for M in (1, 2, 4, 8):
                now = streams(M, N, K, SMS)
                assert now >= before(M, N, K) and (now > 0) == (K <= 338 * 128)
    assert streams(9, 64, 64, SMS) == 0 and streams(0, 64, 64, SMS) == 0

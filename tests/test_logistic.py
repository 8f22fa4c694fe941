"""The logistic function without the division's branch, by way of a convolution of one tap and weight one: 32-bit x / (1 + exp(-x)) against
64 bits over the whole range, and what is no number or infinite where the division would put it."""

import pytest
import torch

from rusty_llama_b200.kernels import ops

pytestmark = pytest.mark.gpu


def _silu(x):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    rows = x.cuda().view(-1, 8)
    one = torch.ones(1, 8, device="cuda")
    seqs = torch.zeros(rows.shape[0], dtype=torch.int32, device="cuda")
    return ops.short_conv(rows, one, None, i32([0]), i32([0, rows.shape[0]]), seqs, silu=True).view(-1).cpu()


@pytest.mark.parametrize("span", [1e-3, 1.0, 20.0, 87.0])
def test_against_64_bits(span):
    x = torch.linspace(-span, span, 1 << 20)
    want = x.double() / (1 + torch.exp(-x.double()))
    # the exponential is two units of 2^-23 off at most, the sum and the quotient half a unit each
    assert bool(((_silu(x).double() - want).abs() <= want.abs() * 6 * 2.0**-24 + 1e-44).all())


def test_beside_the_division():
    """The quotient on its own: the same exponential under the division, one unit in the last place off at most and almost never that, over the
    whole range, for divisors just below and above powers of two and for those whose reciprocal is no normal number."""
    near = torch.tensor([-torch.log(torch.tensor(2.0**k * (1 + e) - 1, dtype=torch.float64)) for k in range(1, 127) for e in torch.linspace(-1e-4, 1e-4, 512, dtype=torch.float64).tolist()])
    x = torch.cat([torch.linspace(-88, 88, 1 << 22), torch.linspace(-1, 1, 1 << 20), near.float(), torch.linspace(-88.72, -87.3, 1 << 16), torch.tensor([2.0**k for k in range(-24, 7)] + [0.0])])
    x = x[: x.numel() // 8 * 8].cuda()
    want, got = x / (1 + torch.exp(-x)), _silu(x).cuda()
    normal = want.abs() > 1.2e-38
    off = (got.view(torch.int32) - want.view(torch.int32)).abs()
    assert int(off[normal].max()) <= 1 and float((off[normal] != 0).double().mean()) <= 1e-6
    assert bool((off[~normal] <= 2).all())


def test_infinities_and_what_is_no_number():
    inf, nan = float("inf"), float("nan")
    x = torch.tensor([inf, -inf, nan, 0.0, 100.0, -100.0, 3e38, -3e38])
    got = _silu(x)
    assert got[0] == inf and got[1].isnan() and got[2].isnan() and got[3] == 0 and got[4] == 100 and got[6] == x[6]
    assert float(got[5].abs()) <= 1e-41 and got[7] == 0

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


def test_infinities_and_what_is_no_number():
    inf, nan = float("inf"), float("nan")
    x = torch.tensor([inf, -inf, nan, 0.0, 100.0, -100.0, 3e38, -3e38])
    got = _silu(x)
    assert got[0] == inf and got[1].isnan() and got[2].isnan() and got[3] == 0 and got[4] == 100 and got[6] == x[6]
    assert float(got[5].abs()) <= 1e-41 and got[7] == 0

"""The causal convolution of long prompts (runs of tokens in registers) against the kernel that takes every token by itself: the same
sums in the same order, so equal bits, whatever the taps, where runs meet the sequences' borders, and in the last, shorter run."""

import pytest
import torch

from rusty_llama_b200.kernels import ops

pytestmark = pytest.mark.gpu


def _i32(a):
    return torch.tensor(a, dtype=torch.int32, device="cuda")


def _conv(x, w, state, slots, lens, bias, silu):
    start = [sum(lens[:i]) for i in range(len(lens) + 1)]
    return ops.short_conv(x, w, state, _i32(slots), _i32(start), _i32([s for s, n in enumerate(lens) for _ in range(n)]), bias=bias, silu=silu)


@pytest.mark.parametrize("taps, bias, silu", [(1, True, True), (2, False, True), (3, True, False), (4, False, True), (4, True, True), (5, False, True)])
@pytest.mark.parametrize("C", [4096, 4104])
def test_runs_equal_tokens_by_themselves(C, taps, bias, silu):
    lens = [300, 3, 1, 2, 7, 297, 1]  # 611 tokens of 512 or 513 threads in a row: runs; the calls below bring too few tokens for them
    g = torch.Generator().manual_seed(C + taps)
    T, wide = sum(lens), C + 24
    x = torch.randn(T, wide, generator=g).to("cuda", torch.bfloat16)[:, 8 : 8 + C]
    w = torch.randn(taps, C, generator=g).cuda()
    b = torch.randn(C, generator=g).cuda() if bias else None
    one = torch.randn(9, taps - 1, C, generator=g).cuda() if taps > 1 else None
    two = one.clone() if taps > 1 else None
    slots = [8, 2, 3, 0, 5, 1, 7]
    got = _conv(x, w, one, slots, lens, b, silu)
    at = 0
    for s, n in enumerate(lens):
        done = 0
        while done < n:
            take = min(n - done, 160)
            rows = slice(at + done, at + done + take)
            assert torch.equal(got[rows], _conv(x[rows], w, two, [slots[s]], [take], b, silu)), (s, done)
            done += take
        at += n
    if taps > 1:
        assert torch.equal(one, two)

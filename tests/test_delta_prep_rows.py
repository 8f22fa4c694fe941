"""The delta rule's unit vectors from rows of whole fours against 64 bits and against the kernel that takes numbers singly (reached here
by rows an odd number apart): keys of a few numbers, of more than 128 and of 256, pairs that do not fill the last block."""

import pytest
import torch

from rusty_llama_b200.kernels import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T, G, H, dim", [(1, 1, 1, 4), (5, 3, 6, 36), (67, 1, 2, 128), (9, 2, 4, 132), (13, 5, 5, 256)])
def test_rows_of_fours_against_64_bits(T, G, H, dim):
    g = torch.Generator().manual_seed(T + dim)
    qk, ba = torch.randn(T, 2 * G * dim, generator=g).to(torch.bfloat16), (2 * torch.randn(T, 2 * H, generator=g)).to(torch.bfloat16)
    a_log, dt_bias = torch.randn(H, generator=g), torch.randn(H, generator=g)
    odd = torch.empty(T, 2 * G * dim + 1, dtype=torch.bfloat16, device="cuda")
    odd[:, :-1] = qk.cuda()
    run = lambda rows: ops.delta_prep(rows, ba.cuda(), a_log.cuda(), dt_bias.cuda(), G, H, dim, 1e-6, dim ** -0.5, log_decay=True)  # noqa: E731
    got, general = run(qk.cuda()), run(odd[:, :-1])
    q, k = qk.double().view(T, 2, G, dim).unbind(1)
    qn, kn = (x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt() for x in (q, k))
    b, a = ba.double().split(H, dim=1)
    log = -a_log.double().exp() * torch.nn.functional.softplus(a + dt_bias.double())
    # a sum of squares is at most 8 numbers and 5 halvings away from its terms, a root and a quotient behind it: 16 roundings; products add
    # up to at most |qn| |kn| = dim^-0.5 with as many again
    unit = 16 * 2.0 ** -24
    want = ((qn * dim ** -0.5).reshape(T, -1), kn.reshape(T, -1), (qn * kn).sum(-1) * dim ** -0.5, b.sigmoid(), log.exp(), log)
    for out in (got, general):
        for name, x, y in zip(("qn", "kn", "kq", "beta", "decay", "log"), out, want):
            size = dim ** -0.5 if name == "kq" else y.abs()
            bound = size * 3 * unit if name != "decay" else size * (log.abs() + 1) * unit
            assert bool(((x.double().cpu() - y).abs() <= bound + 1e-38).all()), name
    for x, y in zip(got[3:], general[3:]):  # the heads' scalars are the same arithmetic
        assert torch.equal(x, y)

"""The chunked walk with a decay per channel on the tensor cores, at sizes where its tiles end: key and value sizes below, at and past a
tile of 16, 64 and 128, heads that share queries and keys, chunks that end inside an eight, and decays from none to ones that underflow
within a few tokens; against 64 bits and beside the FMA kernels, which take the same call with input strengths of one.

Tolerance: the products are exact to 2^-26 and every sum of at most dim + 64 of them is rounded in 32 bits, as in the FMA kernels
(`test_gated_chunk_sizes`): 5e-5 of the largest output holds (dim + 64 + 13) 2^-24 and the state's carry over five chunks."""

import pytest
import torch

from rusty_llama_b200.kernels import ops

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _oracle(q, k, v, a, start, q_scale):
    T, H, dim = k.shape
    out, finals = torch.zeros(T, H, v.shape[2], dtype=F64), []
    for s, e in zip(start[:-1], start[1:]):
        S = torch.zeros(H, dim, v.shape[2], dtype=F64)
        for t in range(s, e):
            S = S * torch.exp(a[t])[:, :, None] + k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hd,hdv->hv", q[t] * q_scale, S)
        finals.append(S)
    return out, torch.stack(finals)


@pytest.mark.parametrize("decay", [0.0, 0.2, 40.0])
@pytest.mark.parametrize("dim, vdim, share", [(8, 8, 1), (24, 72, 2), (64, 64, 1), (72, 104, 1), (120, 128, 2), (128, 128, 1), (128, 136, 1)])
def test_chunked_walk(dim, vdim, share, decay):
    H, start = 2, [0, 17, 18, 18 + 64, 18 + 64 + 305]
    QH, T = H // share, 18 + 64 + 305
    g = torch.Generator().manual_seed(dim * 1000 + vdim)
    rows = torch.randn(T, 2 * QH * dim + H * vdim + 8, generator=g).to(torch.bfloat16)
    proj = rows.cuda()[:, 8:]
    qs, ks, vs = proj[:, : QH * dim], proj[:, QH * dim : 2 * QH * dim], proj[:, 2 * QH * dim :]
    a = (-decay * torch.rand(T, H, dim, generator=g)).float()
    q, k = (x.to(F64).cpu().view(T, QH, dim).repeat_interleave(share, 1) for x in (qs, ks))
    want, final = _oracle(q, k, vs.to(F64).cpu().view(T, H, vdim), a.to(F64), start, 0.25)
    n, slots = len(start) - 1, [4, 0, 3, 2]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731

    def walk(strength):
        state = torch.zeros(n + 1, H, dim, vdim, device="cuda")
        state[1] = 7.0  # a slot of nobody's
        scratch = torch.full((ops.gated_attn_chunked_scratch_floats(n, 305, H, dim, vdim),), float("nan"), device="cuda")
        got = ops.gated_attn_chunked(qs, ks, vs, a.cuda().view(T, -1).contiguous(), strength, state, i32(slots), i32(start), H, dim, vdim, 305, scratch,
                                     q_scale=0.25, qk_heads=QH)
        assert bool((state[1] == 7.0).all())
        return got.view(T, H, vdim).cpu().to(F64), state[slots].cpu().to(F64)

    got, state = walk(None)
    assert float((got - want).abs().max()) <= 5e-5 * float(want.abs().max())
    assert float((state - final).abs().max()) <= 5e-5 * float(final.abs().max())
    other, other_state = walk(torch.ones(T, H, device="cuda"))
    assert float((got - other).abs().max()) <= 1e-4 * float(want.abs().max())
    assert float((state - other_state).abs().max()) <= 1e-4 * float(final.abs().max())


def test_a_value_that_is_no_number_stays_in_its_column_and_its_sixteen():
    H, dim, vdim, T = 1, 64, 64, 130
    g = torch.Generator().manual_seed(5)
    rows = torch.randn(T, 2 * dim + vdim, generator=g).to(torch.bfloat16)
    rows[40, 2 * dim + 3] = float("inf")
    proj = rows.cuda()
    a = (-0.1 * torch.rand(T, H * dim, generator=g)).float().cuda()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    scratch = torch.empty(ops.gated_attn_chunked_scratch_floats(1, T, H, dim, vdim), device="cuda")
    got = ops.gated_attn_chunked(proj[:, :dim], proj[:, dim : 2 * dim], proj[:, 2 * dim :], a, None, torch.zeros(1, H, dim, vdim, device="cuda"), i32([0]),
                                 i32([0, T]), H, dim, vdim, T, scratch)
    bad = ~torch.isfinite(got).cpu()
    assert bool(bad[40:, 3].all()) and not bool(bad[:32].any())
    bad[:, 3] = False
    assert not bool(bad.any())


@pytest.mark.parametrize("dim, vdim, act, off", [(128, 128, 2, 0), (64, 72, 1, 2), (120, 8, 0, 0), (128, 128, None, 0)])
def test_the_norm_taken_along(dim, vdim, act, off):
    """The same sums through the norm inside the kernel and behind it: a rounding of each of two 32-bit chains apart, then rounded to bfloat16
    (2^-8 at most where that falls on different sides)."""
    H, start = 2, [0, 70, 75, 210]
    T = start[-1]
    g = torch.Generator().manual_seed(dim + vdim)
    proj = torch.randn(T, 2 * H * dim + H * vdim, generator=g).to(torch.bfloat16).cuda()
    qs, ks, vs = proj[:, : H * dim], proj[:, H * dim : 2 * H * dim], proj[:, 2 * H * dim :]
    gate = None if act is None else torch.randn(T, off + H * vdim, generator=g).to(torch.bfloat16).cuda()[:, off:]
    a = (-0.2 * torch.rand(T, H * dim, generator=g)).float().cuda()
    w = torch.randn(vdim, generator=g).cuda()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731

    def walk(norm):
        scratch = torch.empty(ops.gated_attn_chunked_scratch_floats(3, 135, H, dim, vdim), device="cuda")
        return ops.gated_attn_chunked(qs, ks, vs, a, None, torch.zeros(3, H, dim, vdim, device="cuda"), i32([0, 1, 2]), i32(start), H, dim, vdim, 135, scratch, norm=norm)

    into = torch.empty(T, H * vdim + 6, dtype=torch.bfloat16, device="cuda")[:, 4 : 4 + H * vdim]
    got = walk((w, 1e-5, gate, act or 0, 0.5, into))
    assert got is into
    want = ops.head_norm_gate(walk(None), H, vdim, w, 1e-5, gate, act or 0, torch.bfloat16, out_scale=0.5)
    assert float(((got.float() - want.float()).abs() / (want.float().abs() + 1e-3)).max()) <= 2.0**-7
    assert float((got != want).float().mean()) <= 0.01
    # rows that start off four bytes: nothing is launched, the caller norms by itself
    odd = torch.empty(T, H * vdim + 1, dtype=torch.bfloat16, device="cuda")[:, 1:]
    assert walk((w, 1e-5, gate, act or 0, 0.5, odd)) is None

"""The chunked walk of a gated recurrence, and the heads' norm behind it, at sizes where their reads change: key and value sizes that
are whole fours and that are not, rows that start off four elements, a last column tile of one to four columns, key sizes around the
128 rows of a pass and the largest that an SM's shared memory takes, heads that share queries and keys, chunk ends inside a sub-chunk.

Tolerance: an output is a sum of at most dim + 64 products, each with a decay whose exponent is a sum of 64 logarithms below 0.2:
(dim + 64 + 13) roundings of 2^-24 in the worst case, 2.2e-5 of the largest sum of magnitudes at dim = 292; 5e-5 of the largest output
holds that and the state's carry over five chunks (random signs keep the errors below the worst case)."""

import pytest
import torch

from rusty_llama_b200.kernels import ops

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _oracle(q, k, v, a, b, start, ext, q_scale):
    T, H, dim = k.shape
    if ext:
        v = torch.cat([v, torch.ones(T, H, 1, dtype=F64)], dim=2)
    out = torch.zeros(T, H, v.shape[2], dtype=F64)
    finals = []
    for s, e in zip(start[:-1], start[1:]):
        S = torch.zeros(H, dim, v.shape[2], dtype=F64)
        for t in range(s, e):
            S = S * torch.exp(a[t])[:, :, None] + (b[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hd,hdv->hv", q[t] * q_scale, S)
        finals.append(S)
    return out, torch.stack(finals)


# key size, value size, normaliser column, per-channel decays, heads per q/k head, elements before the rows
SIZES = [(1, 1, False, True, 1, 0), (3, 5, True, True, 1, 0), (8, 64, False, True, 1, 0), (12, 64, True, False, 1, 0), (30, 63, True, True, 1, 0),
         (64, 68, False, True, 1, 0), (64, 64, False, True, 2, 1), (100, 66, False, False, 2, 0), (124, 128, False, True, 1, 2), (128, 128, False, True, 1, 0),
         (128, 128, True, False, 1, 0), (128, 130, False, True, 1, 4), (132, 32, False, True, 1, 0), (200, 65, False, True, 1, 3), (292, 20, True, True, 1, 0)]


@pytest.mark.parametrize("dim, vdim, ext, channels, share, off", SIZES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_chunked_walk(dtype, dim, vdim, ext, channels, share, off):
    assert ops.gated_attn_chunked_takes(dim, vdim + int(ext)) and not ops.gated_attn_chunked_takes(293, vdim)
    H, start = 2, [0, 17, 18, 18 + 64, 18 + 64 + 305]
    QH, T = H // share, 18 + 64 + 305
    g = torch.Generator().manual_seed(dim * 1000 + vdim)
    wide = 2 * QH * dim + H * vdim
    rows = torch.zeros(T, wide + off + (-(wide + off)) % 4 + (0 if off != 1 else 1), dtype=dtype)
    rows[:, off : off + wide] = torch.randn(T, wide, generator=g).to(dtype)
    proj = rows.cuda()[:, off : off + wide]
    qs, ks, vs = proj[:, : QH * dim], proj[:, QH * dim : 2 * QH * dim], proj[:, 2 * QH * dim :]
    a = (-0.2 * torch.rand(T, H, dim if channels else 1, generator=g)).float()
    b = torch.rand(T, H, generator=g).float()
    q, k = (x.to(F64).cpu().view(T, QH, dim).repeat_interleave(share, 1) for x in (qs, ks))
    want, final = _oracle(q, k, vs.to(F64).cpu().view(T, H, vdim), a.to(F64).expand(T, H, dim), b.to(F64), start, ext, 0.25)
    n, vcols = len(start) - 1, vdim + int(ext)
    state = torch.zeros(n + 1, H, dim, vcols, device="cuda")
    state[1] = 7.0  # a slot of nobody's
    slots = [4, 0, 3, 2]
    scratch = torch.empty(ops.gated_attn_chunked_scratch_floats(n, 305, H, dim, vcols), device="cuda")
    got = ops.gated_attn_chunked(qs, ks, vs, a.cuda().view(T, -1).contiguous(), b.cuda(), state, torch.tensor(slots, dtype=torch.int32, device="cuda"),
                                 torch.tensor(start, dtype=torch.int32, device="cuda"), H, dim, vdim, 305, scratch, q_scale=0.25, ext=ext, qk_heads=QH)
    assert float((got.view(T, H, vcols).cpu().to(F64) - want).abs().max()) <= 5e-5 * float(want.abs().max())
    assert float((state[slots].cpu().to(F64) - final).abs().max()) <= 5e-5 * float(final.abs().max())
    assert bool((state[1] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n, off", [(1, 0), (4, 0), (6, 0), (128, 0), (128, 1), (130, 0), (512, 0), (510, 2)])
def test_head_norm_and_log_decay(dtype, n, off):
    """Outputs are one division, a square root and a logistic away from a sum of at most 512 squares: 1e-5, and the type's rounding."""
    T, H, eps = 37, 3, 1e-5
    g = torch.Generator().manual_seed(n)
    x = torch.randn(T, H * n, generator=g)
    rows = torch.randn(T, off + H * n + (-(off + H * n)) % 4, generator=g).to(dtype)
    gate, w = rows.cuda()[:, off : off + H * n], torch.randn(n, generator=g)
    got = ops.head_norm_gate(x.cuda(), H, n, w.cuda(), eps, gate, ops.GATE_SILU, dtype).to(F64).cpu()
    xd, gd = x.to(F64).view(T, H, n), rows[:, off : off + H * n].to(F64)
    want = (xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + eps) * w.to(F64)).view(T, H * n) * gd * torch.sigmoid(gd)
    room = 2.0**-8 if dtype == torch.bfloat16 else 0.0
    assert bool(((got - want).abs() <= 1e-5 * (1 + want.abs()) + room * want.abs()).all())
    la = ops.gla_log_decay(gate, None, 7.0).to(F64).cpu()
    ref = torch.nn.functional.logsigmoid(gd) / 7.0
    assert float((la - ref).abs().max()) <= 1e-6 * (1 + float(ref.abs().max()))

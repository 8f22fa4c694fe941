"""Which steps of latent attention expand keys and values per head: the work of both forms, counted, and the limit of the bytes.  (The rule
looks at sizes on the host only; the tensors here are stand-ins.)"""

from types import SimpleNamespace

import pytest
import torch

LITE = dict(num_heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512)
SMALL = dict(num_heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256)


def rows(size, pos0, q_lens, window=0, told=True):
    from rusty_llama_b200.parts import MIXERS, Runtime
    from rusty_llama_b200.spec import PartSpec

    part = MIXERS.build(PartSpec("latent_attention", dict(
        size, hidden_size=64, scale=1.0, eps=1e-5, window=window,
        position=PartSpec("rotary", {"rotary_dim": size["rot_dim"], "theta": 1e4, "scaling": None, "interleaved": False}))), Runtime.create("cpu", torch.bfloat16))
    part.w_vk = object()
    q = SimpleNamespace(is_cuda=True, stride=lambda i: 4096, data_ptr=lambda: 0)
    lens = [p + n for p, n in zip(pos0, q_lens)]
    step = SimpleNamespace(decode_only=max(q_lens) == 1, n_tokens=sum(q_lens), n_seqs=len(q_lens), max_q_len=max(q_lens), max_kv_len=max(lens), q_lens=q_lens,
                           pos0=pos0 if told else None)
    got = part._expands(step, q, None)
    assert got in (0, (max(lens) + 63) // 64 * 64)
    return got


@pytest.mark.parametrize("told", [True, False])
@pytest.mark.parametrize("size, pos0, q_lens, window, expands", [
    (LITE, [0], [2048], 0, True),
    (LITE, [0], [33], 0, True),
    (LITE, [0], [32], 0, False),  # (the few-row form of the head products)
    (SMALL, [0, 0, 0, 0], [300, 41, 5, 222], 0, True),
    # a chunk of a prompt onto a long past: every row is seen by every query, and a window cuts that short
    (LITE, [59000], [1024], 0, True),
    (LITE, [59000], [1024], 512, False),
    (LITE, [1000], [1024], 512, True),
    # few queries per row: 41 break even at the larger sizes, 21 at the smaller ones
    (LITE, [2000], [33], 0, False),
    (LITE, [2000], [60], 0, True),
    (SMALL, [2000], [33], 0, True),
])
def test_the_work_decides(size, pos0, q_lens, window, expands, told):
    assert bool(rows(size, pos0, q_lens, window, told)) == expands


def test_long_sequences_that_bring_single_tokens_count_with_their_own_lengths():
    assert not rows(LITE, [0] + [8000] * 8, [2048] + [1] * 8)
    assert rows(LITE, [0] + [200] * 8, [2048] + [1] * 8)
    assert not rows(LITE, [0] + [2000] * 64, [2048] + [1] * 64)


def test_the_limit_counts_the_latents_beside_the_expanded_rows():
    per_row = 2 * (16 * (128 + 128 + 64) + 512)
    most = (1 << 30) // per_row // 64 * 64
    assert rows(LITE, [most - 4096], [4096]) and not rows(LITE, [most - 4095], [4096])

"""What a routed feed-forward holds after loading."""

import torch


def test_a_shared_expert_is_held_once():
    """The experts' matrices and a shared expert's, once each, however steps use them: no copy of it beside the others'."""
    from rusty_llama_b200.parts import FEED_FORWARDS, Runtime
    from rusty_llama_b200.spec import PartSpec

    part = FEED_FORWARDS.build(PartSpec("routed_experts", {"hidden_size": 64, "n_experts": 4, "top": 2, "expert_ff": 32, "bias": False, "renormalize": True,
                                                           "shared_ff": 96, "shared_gate": True}), Runtime.create("cpu", torch.bfloat16))
    w = {name: torch.randn(info.shape).to(torch.float32 if info.kind == "scalars" else torch.bfloat16) for name, info in part.param_infos().items()}
    part.load(w)
    held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for k, t in vars(part).items() if torch.is_tensor(t) and "router" not in k}
    assert sum(held.values()) == sum(2 * t.numel() for t in w.values() if t.dtype == torch.bfloat16)
    assert part.always == 3
    for j in range(3):  # the pieces of it that steps of few tokens send along with the experts
        assert torch.equal(part.always_gate[j], w["shared.gate"][32 * j : 32 * j + 32]) and torch.equal(part.always_up[j], w["shared.up"][32 * j : 32 * j + 32])
        assert torch.equal(part.always_down[j], w["shared.down"][:, 32 * j : 32 * j + 32])

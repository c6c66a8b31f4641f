"""The state of a decode step, which the kernels read and write where it lies."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _token(B, H, K, V, T=1):
    gen = torch.Generator(device="cuda").manual_seed(9)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    return dict(q=r(B, T, H, K), k=r(B, T, H, K) / K ** 0.5, v=r(B, T, H, V), g=-r(B, T, H, K).abs() / 16, beta=r(B, T, H).sigmoid())


def _step(op, x, state):
    from tops_b200.ops.gla import fused_recurrent_gla_decode_
    from tops_b200.ops.kda import fused_recurrent_kda_decode_
    if op == "kda":
        return fused_recurrent_kda_decode_(x["q"], x["k"], x["v"], x["g"], x["beta"], state)
    return fused_recurrent_gla_decode_(x["q"], x["k"], x["v"], x["g"], state)


@pytest.mark.parametrize("op", ["gla", "kda"])
def test_a_state_that_is_not_on_the_gpu_is_refused(op):
    x = _token(1, 2, 64, 64)
    with pytest.raises(AssertionError):
        _step(op, x, torch.zeros(1, 2, 64, 64))

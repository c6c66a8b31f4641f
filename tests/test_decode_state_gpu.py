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


@pytest.mark.parametrize("offset", [1, 2, 4])
@pytest.mark.parametrize("op,T,K,V", [("gla", 1, 128, 128), ("gla", 3, 64, 36), ("kda", 1, 128, 128), ("kda", 16, 64, 64), ("kda", 1, 200, 256)])
def test_a_state_at_any_offset_of_a_cache(op, T, K, V, offset):
    """A contiguous view into a larger cache starts on no 16-byte boundary: the state goes element by element then."""
    B, H = 2, 3
    x = _token(B, H, K, V, T)
    n = B * H * K * V
    cache = torch.randn(n + 8, device="cuda")
    aligned = cache[offset:offset + n].clone().view(B, H, K, V)
    before = cache.clone()
    view = cache[offset:offset + n].view(B, H, K, V)
    assert (view.data_ptr() % 16 == 0) == (offset == 4)
    want = _step(op, x, aligned)
    got = _step(op, x, view)
    assert torch.equal(got, want) and torch.equal(view, aligned)
    assert torch.equal(cache[:offset], before[:offset]) and torch.equal(cache[offset + n:], before[offset + n:])


@pytest.mark.parametrize("op", ["gla", "kda"])
def test_an_initial_state_at_any_offset(op):
    from tops_b200.ops.gla import fused_recurrent_gla
    from tops_b200.ops.kda import fused_recurrent_kda
    x = _token(1, 2, 64, 64, 5)
    h0 = torch.randn(2 * 64 * 64 + 1, device="cuda")[1:].view(1, 2, 64, 64)
    run = (lambda h: fused_recurrent_kda(x["q"], x["k"], x["v"], x["g"], x["beta"], initial_state=h, output_final_state=True)) if op == "kda" \
        else (lambda h: fused_recurrent_gla(x["q"], x["k"], x["v"], x["g"], initial_state=h, output_final_state=True))
    for a, b in zip(run(h0), run(h0.clone())):
        assert torch.equal(a, b)

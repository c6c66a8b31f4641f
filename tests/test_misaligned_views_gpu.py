"""Contiguous views that start on no 16-byte boundary of a larger tensor: time slices of packed projections and gates."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(t):
    """The same values two or four bytes past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = flat[1:].view(t.shape)
    view.copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16 != 0
    return view


def _same(a, b):
    """Equal but for the order of a few fp32 additions (sums of a scalar gate's gradient and of dbeta over channels): those of
    n terms differ by less than n 2^-24 of their absolute sum, and by one unit of the result's own type."""
    assert (a.double() - b.double()).norm() <= (2 ** -8 if a.dtype == torch.bfloat16 else 1e-5) * b.double().norm()
    assert (a != b).double().mean() <= 0.01 or a.dtype == torch.float32


def _draw(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def _inputs(B, T, H, K, V, dtype, scalar):
    d = lambda i, *s: _draw(*s, seed=i).to(dtype)
    return [d(0, B, T, H, K), d(1, B, T, H, K), d(2, B, T, H, V), -(_draw(B, T, H, seed=3) if scalar else _draw(B, T, H, K, seed=3)).abs().to(dtype) / 16,
            _draw(B, H, K, V, seed=4), d(5, B, T, H, V), _draw(B, H, K, V, seed=6)]


@pytest.mark.parametrize("op", ["chunk_gla", "chunk_simple_gla", "kda", "fused_recurrent_gla"])
@pytest.mark.parametrize("T,K,dtype", [(100, 128, torch.bfloat16), (64, 128, torch.bfloat16), (70, 64, torch.float32)])
def test_ops(op, T, K, dtype):
    from tops_b200.ops.gla import chunk_gla, fused_recurrent_gla
    from tops_b200.ops.kda import chunk_kda, fused_recurrent_kda
    from tops_b200.ops.simple_gla import chunk_simple_gla
    q, k, v, g, h0, do, dht = _inputs(1, T, 2, K, K, dtype, op == "chunk_simple_gla")
    beta = _draw(1, T, 2, seed=7).sigmoid().to(dtype)
    k = k / K ** 0.5
    run = {"chunk_gla": lambda *a: chunk_gla(*a[:4], initial_state=a[4], output_final_state=True),
           "chunk_simple_gla": lambda *a: chunk_simple_gla(*a[:3], g=a[3], initial_state=a[4], output_final_state=True),
           "kda": lambda *a: (chunk_kda if T % 64 == 0 else fused_recurrent_kda)(*a[:4], beta, initial_state=a[4], output_final_state=True),
           "fused_recurrent_gla": lambda *a: fused_recurrent_gla(*a[:4], initial_state=a[4], output_final_state=True)}[op]
    results = []
    for place in (lambda t: t.clone(), _off):
        leaves = [place(t).requires_grad_() for t in (q, k, v, g, h0)]
        o, ht = run(*leaves)
        results.append([o, ht, *torch.autograd.grad([o, ht], leaves, [place(do), place(dht)])])
    for a, b in zip(*results):
        _same(a, b)


def test_explicit_backward_and_a_time_slice_of_scalar_gates():
    from tops_b200.ops.gla import chunk_gla_bwd
    from tops_b200.ops.simple_gla import chunk_simple_gla, chunk_simple_gla_bwd
    q, k, v, g, h0, do, dht = _inputs(1, 100, 3, 64, 64, torch.bfloat16, False)
    for a, b in zip(chunk_gla_bwd(q, k, v, g, None, 0.1, h0, None, None, do, dht),
                    chunk_gla_bwd(*map(_off, (q, k, v, g)), None, 0.1, _off(h0), None, None, _off(do), _off(dht))):
        assert torch.equal(a, b)
    s = -_draw(1, 131, 4, seed=8).abs().to(torch.bfloat16) / 16
    part = s[:, 31:]
    q, k, v = (_draw(1, 100, 4, 128, seed=i).to(torch.bfloat16) for i in range(3))
    assert part.is_contiguous() and part.data_ptr() % 16 != 0
    assert torch.equal(chunk_simple_gla(q, k, v, g=part)[0], chunk_simple_gla(q, k, v, g=part.clone())[0])
    for a, b in zip(chunk_simple_gla_bwd(q, k, v, part, None, None, v, None, 0.1), chunk_simple_gla_bwd(q, k, v, part.clone(), None, None, v, None, 0.1)):
        assert a is b is None or _same(a, b) is None


def test_gates_norms_and_the_layer():
    from tops_b200.layers import GatedLinearAttention
    from tops_b200.ops.gate import gla_gate, kda_gate_fwd
    from tops_b200.ops.norm import l2norm, rmsnorm_gated
    x, A, b, w = _draw(2, 9, 4, 64).to(torch.bfloat16), _draw(4, seed=1), _draw(256, seed=2), _draw(64, seed=3)
    for f in (gla_gate, l2norm, lambda t: kda_gate_fwd(t, A, _off(b)), lambda t: rmsnorm_gated(t, t, _off(w))):
        assert torch.equal(f(x), f(_off(x)))
    layer = GatedLinearAttention(hidden_size=256, num_heads=2).cuda().to(torch.bfloat16)
    with torch.no_grad():
        for T in (1, 80):
            x = _draw(1, T, 256, seed=T).to(torch.bfloat16)
            assert torch.equal(layer(x)[0], layer(_off(x))[0])
        want = layer(x)[0].double()
        layer.q_proj.weight.data = _off(layer.q_proj.weight.data)
        layer.gk_proj[1].bias.data = _off(layer.gk_proj[1].bias.data)
        got = layer(x)[0].double()   # (through the modules: other roundings)
        assert ((got - want).norm() / want.norm()).item() <= 1e-2

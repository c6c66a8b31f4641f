"""The ops under `torch.jit.trace` and under forward-mode differentiation, where a node made in C++ would be passed by."""
import pytest
import torch
from torch.autograd import forward_ad as fwAD


def test_recorded_call_of_any_op():
    """On the CPU, with an op that allocates where a trace does not see it."""
    from tops_b200.ops import _recorded as R

    def op(x, n, y):
        out = torch.empty(3)
        out.data.copy_(x.detach() * n + (0 if y is None else y.detach()))
        return (out, None) if not x.requires_grad else (x * n, None)

    x = torch.ones(3)
    traced = torch.jit.trace(lambda t: R.call(op, t, 3.0, None)[0] + 1, (x,), check_trace=False)
    assert torch.equal(traced(2 * x), torch.full((3,), 7.0))
    leaf = x.clone().requires_grad_()
    torch.jit.trace(lambda t: R.call(op, t, 3.0, None)[0], (leaf,), check_trace=False)(leaf).sum().backward()
    assert torch.equal(leaf.grad, torch.full((3,), 3.0))
    with fwAD.dual_level(), pytest.raises(NotImplementedError):
        R.call(op, fwAD.make_dual(x, x), 3.0, None)
    assert R.call(op, x, 3.0, x)[0].tolist() == [4.0] * 3


def _ops():
    from tops_b200.ops.gate import gla_gate, kda_gate_fwd
    from tops_b200.ops.gla import chunk_gla, fused_recurrent_gla
    from tops_b200.ops.kda import chunk_kda, fused_recurrent_kda
    from tops_b200.ops.norm import l2norm, rmsnorm_gated
    from tops_b200.ops.simple_gla import chunk_simple_gla
    A = torch.zeros(2, device="cuda")
    return {
        "chunk_gla": lambda x: chunk_gla(x, x, x, -x.abs(), output_final_state=True)[0],
        "chunk_simple_gla": lambda x: chunk_simple_gla(x, x, x, g=-x[..., 0].abs())[0],
        "fused_recurrent_gla": lambda x: fused_recurrent_gla(x, x, x, -x.abs())[0],
        "chunk_kda": lambda x: chunk_kda(x, x, x, -x.abs(), x[..., 0].sigmoid())[0],
        "fused_recurrent_kda": lambda x: fused_recurrent_kda(x, x, x, -x.abs(), x[..., 0].sigmoid())[0],
        "kda_gate": lambda x: kda_gate_fwd(x, A), "gla_gate": gla_gate, "l2norm": l2norm, "rmsnorm_gated": lambda x: rmsnorm_gated(x, x),
    }


NAMES = ["chunk_gla", "chunk_simple_gla", "fused_recurrent_gla", "chunk_kda", "fused_recurrent_kda", "kda_gate", "gla_gate", "l2norm",
         "rmsnorm_gated"]


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_ops(name):
    op = _ops()[name]
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, y = (0.1 * torch.randn(1, 64, 2, 128, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    traced = torch.jit.trace(op, (x,), check_trace=False)
    assert torch.equal(traced(y), op(y))
    with fwAD.dual_level(), pytest.raises(NotImplementedError):
        op(fwAD.make_dual(x, x))
    leaf = y.clone().requires_grad_()
    want = torch.autograd.grad(op(leaf), leaf, x.to(op(y).dtype))[0]
    got = torch.autograd.grad(traced(leaf), leaf, x.to(op(y).dtype))[0]
    assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [3, 80])
def test_layer(T):
    from tops_b200.layers import GatedLinearAttention
    layer = GatedLinearAttention(hidden_size=256, num_heads=2).cuda().to(torch.bfloat16)
    first = torch.nn.Module()
    first.layer = layer
    first.forward = lambda t: layer(t)[0]
    gen = torch.Generator(device="cuda").manual_seed(2)
    x, y = (torch.randn(2, T, 256, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    with torch.no_grad():
        traced = torch.jit.trace(first, (x,), check_trace=False)
        got, want = traced(y).double(), layer(y)[0].double()
        assert ((got - want).norm() / want.norm()).item() <= 1e-2   # (modules against the one call: other roundings)
        with fwAD.dual_level(), pytest.raises(NotImplementedError):
            layer(fwAD.make_dual(x, x))

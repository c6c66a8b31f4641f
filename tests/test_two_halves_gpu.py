"""Precision of the general tcgen05 GLA kernels, whose gated operands and intra-chunk matrices are two bf16 halves each,
against the oracle in fp64."""
import pytest
import torch

from oracle import gla as O
from oracle import simple_gla as OS
from tests.util import rel_l2
from tops_b200.synth import make_inputs

pytestmark = pytest.mark.gpu

# U: the largest relative error of one rounding to bf16.  A result is rounded once, and its inter-chunk part (a fraction
# of it under these gates, all of it at worst) comes from two more roundings, of the chunk-start state and of the operand
# that meets it; roundings are independent, so three of them stay below sqrt(3) U and one and a fraction below 1.25 U.
# Operands or matrices rounded to bf16 inside the chunk give 1.65 U.
U = 2.0 ** -9


def _inputs(seed, B, T, H, D, N, scalar):
    x = make_inputs(seed, B, T, H, D, D, dtype=torch.bfloat16, gate="scalar" if scalar else "per_channel", with_grads=True)
    gen = torch.Generator().manual_seed(seed)
    x["h0"] = 0.1 * torch.randn(N, H, D, D, generator=gen)
    x["dht"] = 0.1 * torch.randn(N, H, D, D, generator=gen)
    return x, {n: t.double() for n, t in x.items()}


def _grads(fn, x, names):
    c = {n: t.cuda() for n, t in x.items()}
    leaves = [c[n].requires_grad_() for n in names]
    o, ht = fn(c)
    return [o, ht, *torch.autograd.grad([o, ht], leaves, [c["do"], c["dht"]])]


@pytest.mark.parametrize("B,T,H,D,cu", [(1, 65, 1, 128, None), (2, 127, 2, 128, None), (1, 1000, 2, 128, None),
                                        (1, 200, 2, 64, None), (1, 300, 2, 128, [0, 1, 64, 129, 300]), (1, 1500, 2, 64, [0, 1300, 1500])])
def test_per_channel_gate(B, T, H, D, cu):
    from tops_b200.ops.gla import chunk_gla
    x, e = _inputs(81, B, T, H, D, B if cu is None else len(cu) - 1, False)
    got = _grads(lambda c: chunk_gla(c["q"], c["k"], c["v"], c["g"], initial_state=c["h0"], output_final_state=True, cu_seqlens=cu),
                 x, ("q", "k", "v", "g", "h0"))
    want = [*O.chunk_gla(e["q"], e["k"], e["v"], e["g"], D ** -0.5, e["h0"], True, cu_seqlens=cu, chunk_size=64),
            *O.chunk_gla_bwd(e["q"], e["k"], e["v"], e["g"], None, D ** -0.5, e["h0"], None, None, e["do"], e["dht"], chunk_size=64,
                             cu_seqlens=cu)]
    for n, a, b in zip(("o", "ht", "dq", "dk", "dv", "dg", "dh0"), got, want):
        # (fp32 states: 2^-17 of what two halves leave out; dh0 comes from one rounded operand)
        bar = 2.0 ** -16 if n == "ht" else 1.25 * U
        assert rel_l2(a, b) <= bar, (n, rel_l2(a, b))


@pytest.mark.parametrize("gate", ["g", "gamma"])
@pytest.mark.parametrize("B,T,H,cu", [(2, 127, 2, None), (1, 1000, 2, None), (1, 300, 2, [0, 1, 64, 129, 300])])
def test_scalar_gate(B, T, H, cu, gate):
    from tops_b200.ops.simple_gla import chunk_simple_gla
    x, e = _inputs(82, B, T, H, 128, B if cu is None else len(cu) - 1, True)
    gamma = -torch.linspace(0.01, 0.2, H) if gate == "gamma" else None
    names = ("q", "k", "v", "g", "h0") if gate == "g" else ("q", "k", "v", "h0")
    gam = None if gamma is None else gamma.cuda()
    got = _grads(lambda c: chunk_simple_gla(c["q"], c["k"], c["v"], c["g"] if gate == "g" else None, gam, None, c["h0"], True,
                                            cu_seqlens=cu), x, names)
    g = e["g"] if gate == "g" else None
    gd = None if gamma is None else gamma.double()
    want = [*OS.chunk_simple_gla(e["q"], e["k"], e["v"], g, gd, 128 ** -0.5, e["h0"], True, cu_seqlens=cu, chunk_size=64)]
    grads = OS.chunk_simple_gla_bwd(e["q"], e["k"], e["v"], g, gd, e["h0"], e["do"], e["dht"], 128 ** -0.5, chunk_size=64, cu_seqlens=cu)
    want += [t for n, t in zip(("q", "k", "v", "g", "h0"), grads) if n in names]
    for n, a, b in zip(("o", "ht", *("d" + n for n in names)), got, want):
        bar = 2.0 ** -16 if n == "ht" else 3 ** 0.5 * U
        assert rel_l2(a, b) <= bar, (n, rel_l2(a, b))

"""Gates that decay a channel by more than fp32 can hold over a chunk: the general tcgen05 GLA kernels against the oracle in
fp64.  Chunks in which some channel's gates sum beyond the kernels' span take another way through them."""
import copy

import pytest
import torch

from oracle import gla as O
from oracle import simple_gla as OS
from tests.util import assert_close, rel_l2

pytestmark = pytest.mark.gpu

CASES = [
    # B, T, H, K, V, cu_seqlens
    (1, 65, 1, 128, 128, None),
    (2, 100, 3, 64, 64, None),
    (1, 1000, 2, 128, 128, None),                      # runs of a cut sequence
    (1, 704, 2, 128, 128, None),                       # whole chunks, a prime number of them
    (1, 130, 2, 128, 256, None),                       # two value slices
    (1, 96, 1, 72, 40, None),
    (1, 300, 2, 128, 128, [0, 1, 64, 129, 300]),
    (1, 1500, 2, 64, 64, [0, 1300, 1500]),
]


def _gates(kind, shape, gen):
    """`mixed`: weak and strong channels side by side, changing from stretch to stretch; `edge`: sums around the limit."""
    if isinstance(kind, float):
        return torch.full(shape, kind)
    if kind == "edge":
        return -2.0 + 0.1 * torch.randn(shape, generator=gen)
    B, T = shape[:2]
    level = torch.tensor([-0.02, -0.5, -3.0, -12.0])[torch.randint(4, (B, (T + 39) // 40, *shape[2:]), generator=gen)]
    return level.repeat_interleave(40, 1)[:, :T] * (0.5 + torch.rand(shape, generator=gen))


def _inputs(seed, B, T, H, K, V, N, kind, scalar):
    gen = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16)
    x = dict(q=r(B, T, H, K), k=r(B, T, H, K), v=r(B, T, H, V), do=r(B, T, H, V),
             h0=torch.randn(N, H, K, V, generator=gen), dht=torch.randn(N, H, K, V, generator=gen))
    x["g"] = _gates(kind, (B, T, H) if scalar else (B, T, H, K), gen).to(torch.bfloat16)
    return x, {n: t.double() for n, t in x.items()}


def _check(run, x, names, want):
    from tops_b200 import _lib as L
    c = {n: t.cuda() for n, t in x.items()}
    leaves = [c[n].requires_grad_() for n in names]
    o, ht = run(c)
    got = [o, ht, *torch.autograd.grad([o, ht], leaves, [c["do"], c["dht"]])]
    assert L.device_error() == 0
    for n, a, b in zip(("o", "ht", *("d" + n for n in names)), got, want):
        assert_close(n, a, b, torch.bfloat16)
        if n not in ("dg", "ht"):   # (three bf16 roundings; dg is what is left of terms that cancel)
            assert rel_l2(a, b) <= 3 ** 0.5 * 2.0 ** -9, (n, rel_l2(a, b))


@pytest.mark.parametrize("kind", [-2.9, -5.0, -11.0, "mixed", "edge"])
@pytest.mark.parametrize("B,T,H,K,V,cu", CASES)
def test_per_channel_gate(B, T, H, K, V, cu, kind):
    from tops_b200.ops.gla import chunk_gla
    x, e = _inputs(91, B, T, H, K, V, B if cu is None else len(cu) - 1, kind, False)
    want = [*O.chunk_gla(e["q"], e["k"], e["v"], e["g"], K ** -0.5, e["h0"], True, cu_seqlens=cu, chunk_size=16),
            *O.chunk_gla_bwd(e["q"], e["k"], e["v"], e["g"], None, K ** -0.5, e["h0"], None, None, e["do"], e["dht"], chunk_size=16,
                             cu_seqlens=cu)]
    _check(lambda c: chunk_gla(c["q"], c["k"], c["v"], c["g"], initial_state=c["h0"], output_final_state=True, cu_seqlens=cu),
           x, ("q", "k", "v", "g", "h0"), want)


@pytest.mark.parametrize("gate", ["g", "gamma"])
@pytest.mark.parametrize("B,T,H,K,V,cu", [CASES[i] for i in (1, 2, 4, 6)])
def test_scalar_gate(B, T, H, K, V, cu, gate):
    from tops_b200.ops.simple_gla import chunk_simple_gla
    x, e = _inputs(92, B, T, H, K, V, B if cu is None else len(cu) - 1, "mixed", True)
    gamma = -torch.tensor([4.0, 0.05, 11.0])[:H] if gate == "gamma" else None
    names = ("q", "k", "v", "g", "h0") if gate == "g" else ("q", "k", "v", "h0")
    g, gd = (e["g"], None) if gate == "g" else (None, gamma.double())
    want = [*OS.chunk_simple_gla(e["q"], e["k"], e["v"], g, gd, K ** -0.5, e["h0"], True, cu_seqlens=cu, chunk_size=16)]
    grads = OS.chunk_simple_gla_bwd(e["q"], e["k"], e["v"], g, gd, e["h0"], e["do"], e["dht"], K ** -0.5, chunk_size=16, cu_seqlens=cu)
    want += [t for n, t in zip(("q", "k", "v", "g", "h0"), grads) if n in names]
    gam = None if gamma is None else gamma.cuda()
    _check(lambda c: chunk_simple_gla(c["q"], c["k"], c["v"], c["g"] if gate == "g" else None, gam, None, c["h0"], True,
                                      cu_seqlens=cu), x, names, want)


def test_a_layer_with_strong_gates():
    from tops_b200.layers import Cache, GatedLinearAttention
    torch.manual_seed(3)
    layer = GatedLinearAttention(hidden_size=512, num_heads=4, layer_idx=0, gate_logit_normalizer=0.15).cuda().to(torch.bfloat16)
    ref = copy.deepcopy(layer).float()
    x = torch.randn(2, 200, 512, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        caches = Cache(), Cache()
        o, want = layer(x, past_key_values=caches[0], use_cache=True)[0], ref(x.float(), past_key_values=caches[1], use_cache=True)[0]
        assert rel_l2(o, want) <= 2e-2 and rel_l2(caches[0][0]["recurrent_state"], caches[1][0]["recurrent_state"]) <= 2e-2
    leaf = x.clone().requires_grad_()
    grads = torch.autograd.grad(layer(leaf)[0].float().square().sum(), [leaf, *layer.parameters()])
    assert all(torch.isfinite(t.float()).all() for t in grads)


@pytest.mark.parametrize("level", [-0.05, -5.0])
def test_a_captured_step(level):
    """Forward + backward of a packed batch in a CUDA graph, replayed on other inputs."""
    from tops_b200.ops.gla import chunk_gla
    cu = [0, 70, 300]
    x, _ = _inputs(93, 1, 300, 2, 128, 128, 2, level, False)
    y, _ = _inputs(94, 1, 300, 2, 128, 128, 2, level, False)
    names = ("q", "k", "v", "g", "h0")
    c = {n: t.cuda() for n, t in x.items()}
    leaves = [c[n].requires_grad_() for n in names]

    def step():
        o, ht = chunk_gla(*leaves[:4], initial_state=leaves[4], output_final_state=True, cu_seqlens=cu)
        return [o, ht, *torch.autograd.grad([o, ht], leaves, [c["do"], c["dht"]])]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    with torch.no_grad():
        for n in c:
            c[n].copy_(y[n])
    graph.replay()
    torch.cuda.synchronize()
    want = step()
    for a, b in zip(captured, want):
        assert torch.equal(a, b)

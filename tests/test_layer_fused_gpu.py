"""`GatedLinearAttention` as one call (bf16) against the same weights run module by module in fp32, and the few-row
projection kernel against torch, at the sizes where they switch form."""
import copy

import pytest
import torch

from tests.util import rel_l2

pytestmark = pytest.mark.gpu


def _layer(hidden, heads, **kw):
    from tops_b200.layers import GatedLinearAttention
    torch.manual_seed(3)
    return GatedLinearAttention(hidden_size=hidden, num_heads=heads, layer_idx=0, **kw).cuda().to(torch.bfloat16)


def _labels(fn):
    import ctypes

    from tops_b200 import _lib as L
    L.lib.tops_b200_profile_enable(1)
    out = fn()
    torch.cuda.synchronize()
    L.lib.tops_b200_profile_enable(0)
    buf = ctypes.create_string_buffer(4096)
    L.lib.tops_b200_profile_read(buf, len(buf))
    return out, [ln.split()[0] for ln in buf.value.decode().splitlines()]


@pytest.mark.parametrize("B,T,hidden,heads,cu", [(2, 65, 512, 4, None), (1, 200, 1024, 4, [0, 70, 71, 200]), (2, 128, 256, 2, None)])
def test_training_step(B, T, hidden, heads, cu):
    layer = _layer(hidden, heads)
    ref = copy.deepcopy(layer).float()
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(B, T, hidden, generator=gen, device="cuda").to(torch.bfloat16)
    do = torch.randn(B, T, hidden, generator=gen, device="cuda").to(torch.bfloat16)

    def run(m, dt):
        leaf = x.to(dt).requires_grad_()
        o = m(leaf, cu_seqlens=cu)[0]
        return [o, *torch.autograd.grad(o, [leaf, *m.parameters()], do.to(dt))]
    got, labels = _labels(lambda: run(layer, torch.bfloat16))
    assert "lowrank_gate_fwd" in labels
    names = ["o", "x", *(n for n, _ in layer.named_parameters())]
    for n, a, b in zip(names, got, run(ref, torch.float32)):
        assert a.dtype == torch.bfloat16 and a.shape == b.shape
        # dq and dk (and so dx) of a sequence's first token are what is left of do . o / |o|^2 after the norm's
        # projection: rounding noise of do, amplified; everything else keeps the bf16 bar (test_training_step_from_a_state
        # holds these three to it too)
        bar = 0.2 if n in ("x", "q_proj.weight", "k_proj.weight") else 2e-2
        assert rel_l2(a, b) <= bar, (n, rel_l2(a, b))


@pytest.mark.parametrize("T,kw,frozen", [(65, {}, ()), (130, {"clamp_min": -0.06}, ()), (100, {"elementwise_affine": False}, ()),
                                         (70, {}, ("q_proj", "gk_proj.0", "o_proj")), (70, {}, ("k_proj", "gk_proj.1", "g_norm_swish_gate"))])
def test_training_step_from_a_state(T, kw, frozen):
    """Every gradient of the one-call layer, the initial state's among them, with a cotangent on the final state.  From a state
    no output is a multiple of one token's v, so no gradient is noise and all keep the bf16 bar.  (The clip takes the tail of
    the gates: one that took half of them would have many at its edge, where a rounding decides about a gradient.)"""
    from tops_b200.layers import Cache
    layer = _layer(512, 4, **kw)
    for n, p in layer.named_parameters():
        p.requires_grad_(not n.startswith(frozen) if frozen else True)
    ref = copy.deepcopy(layer).float()
    gen = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(2, T, 512, generator=gen, device="cuda").to(torch.bfloat16)
    do = torch.randn(2, T, 512, generator=gen, device="cuda").to(torch.bfloat16)
    h0, dht = (torch.randn(2, 4, 64, 128, generator=gen, device="cuda") for _ in range(2))

    def run(m, dt):
        leaf, state, cache = x.to(dt).requires_grad_(), h0.clone().requires_grad_(), Cache()
        cache.update(recurrent_state=state, layer_idx=0)
        o, _, cache = m(leaf, past_key_values=cache, use_cache=True)
        params = [p for p in m.parameters() if p.requires_grad]
        return [o, cache[0]["recurrent_state"], *torch.autograd.grad([o, cache[0]["recurrent_state"]], [leaf, state, *params], [do.to(dt), dht])]
    got, labels = _labels(lambda: run(layer, torch.bfloat16))
    assert "lowrank_gate_fwd" in labels
    names = ["o", "ht", "x", "h0", *(n for n, p in layer.named_parameters() if p.requires_grad)]
    for n, a, b in zip(names, got, run(ref, torch.float32)):
        assert a.shape == b.shape and rel_l2(a, b) <= 2e-2, (n, rel_l2(a, b))


@pytest.mark.parametrize("T1", [1, 3, 64, 65, 130])
@pytest.mark.parametrize("B,hidden,heads", [(1, 1024, 4), (9, 512, 4)])
def test_prompt_then_tokens(B, hidden, heads, T1):
    from tops_b200.layers import Cache
    layer = _layer(hidden, heads, clamp_min=-0.2)
    ref = copy.deepcopy(layer).float()
    gen = torch.Generator(device="cuda").manual_seed(5)
    xs = [torch.randn(B, T, hidden, generator=gen, device="cuda").to(torch.bfloat16) for T in (T1, 1, 2)]
    with torch.no_grad():
        caches = Cache(), Cache()
        for x in xs:
            (o, _, _), labels = _labels(lambda: layer(x, past_key_values=caches[0], use_cache=True))
            assert ("lowrank_gate_fwd" in labels) == (x.shape[1] > 64 or B * x.shape[1] <= 64)
            want = ref(x.float(), past_key_values=caches[1], use_cache=True)[0]
            assert rel_l2(o, want) <= 2e-2
            assert rel_l2(caches[0][0]["recurrent_state"], caches[1][0]["recurrent_state"]) <= 2e-2


def test_watched_or_replaced_projections_are_called():
    layer = _layer(512, 4)
    x = torch.randn(1, 70, 512, device="cuda", dtype=torch.bfloat16)
    seen = []
    handle = layer.o_proj.register_forward_hook(lambda *a: seen.append(1))
    layer(x)
    handle.remove()
    layer.v_proj = torch.nn.Sequential(layer.v_proj)   # no longer a plain linear
    _, labels = _labels(lambda: layer(x))
    assert seen and "lowrank_gate_fwd" not in labels


@pytest.mark.parametrize("T", [1, 70])
@pytest.mark.parametrize("change", ["norm", "gate", "one gate module", "forward", "norm forward", "norm hook"])
def test_any_changed_submodule_is_called(T, change):
    from torch import nn
    layer = _layer(512, 4)
    x = torch.randn(1, T, 512, device="cuda", dtype=torch.bfloat16)
    seen = []

    def wrap(m):
        inner = m.forward
        m.forward = lambda *a: seen.append(1) or inner(*a)

    class Watch(nn.Module):
        def __init__(self, inner=None):
            super().__init__()
            self.inner = inner

        def forward(self, *a):
            seen.append(1)
            return a[0] if self.inner is None else self.inner(*a)
    if change == "norm":
        layer.g_norm_swish_gate = Watch(layer.g_norm_swish_gate)
    elif change == "gate":
        layer.gk_proj.append(Watch())
    elif change == "one gate module":
        layer.gk_proj = Watch(nn.Linear(512, 256, device="cuda", dtype=torch.bfloat16))
    elif change == "norm hook":
        layer.g_norm_swish_gate.register_forward_hook(lambda *a: seen.append(1))
    else:
        wrap(layer.o_proj if change == "forward" else layer.g_norm_swish_gate)
    with torch.no_grad():
        layer(x)
    assert seen


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 16, 31, 33, 64])
@pytest.mark.parametrize("K,Ns", [(32, (8,)), (96, (17, 16, 1)), (2048, (512, 40))])
def test_skinny_linear(rows, K, Ns):
    import ctypes as C

    from tops_b200 import _lib as L
    gen = torch.Generator(device="cuda").manual_seed(rows * K)
    x = torch.randn(rows, K, generator=gen, device="cuda").to(torch.bfloat16)
    Ws = [torch.randn(n, K, generator=gen, device="cuda").to(torch.bfloat16) for n in Ns]
    ys = [torch.full((rows, n + 3), 7.0, device="cuda", dtype=torch.bfloat16) for n in Ns]

    class Params(C.Structure):
        _fields_ = [("rows", C.c_int32), ("K", C.c_int32), ("count", C.c_int32), ("x_pitch", C.c_int64), ("x", C.c_void_p),
                    ("W", C.c_void_p * 6), ("y", C.c_void_p * 6), ("N", C.c_int32 * 6), ("y_pitch", C.c_int64 * 6)]
    p = Params(rows, K, len(Ns), K, x.data_ptr())
    for i, (W, y, n) in enumerate(zip(Ws, ys, Ns)):
        p.W[i], p.y[i], p.N[i], p.y_pitch[i] = W.data_ptr(), y.data_ptr(), n, n + 3
    L.check(L.lib.tops_b200_skinny_linear(C.byref(p), C.c_void_p(L.stream_ptr(x.device))), "skinny_linear")
    for W, y, n in zip(Ws, ys, Ns):
        want = x.double() @ W.double().t()
        # fp32 sums of K products, one rounding to bf16 (2^-9 of the value)
        bar = want.abs() * 2 ** -8 + (x.double().abs() @ W.double().abs().t()) * K * 2 ** -24
        assert ((y[:, :n].double() - want).abs() <= bar).all() and (y[:, n:] == 7).all()


@pytest.mark.parametrize("T", [1, 70])
@pytest.mark.parametrize("change", ["wide", "narrow", "bias", "o_proj", "k_proj", "norm"])
def test_what_does_not_fit_is_refused(T, change):
    """Inputs and weights whose shapes or types do not belong together go through the modules, which refuse them."""
    from torch import nn
    layer = _layer(512, 4)
    hid = {"wide": 544, "narrow": 480}.get(change, 512)
    new = lambda i, o, **kw: nn.Linear(i, o, bias=False, device="cuda", dtype=torch.bfloat16, **kw)
    if change == "bias":
        layer.gk_proj[1].bias.data = layer.gk_proj[1].bias.data.float()
    elif change == "o_proj":
        layer.o_proj = new(544, 512)
    elif change == "k_proj":
        layer.k_proj = new(512, 288)
    elif change == "norm":
        layer.g_norm_swish_gate.weight.data = torch.ones(64, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(2, T, hid, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad(), pytest.raises((RuntimeError, AssertionError)):
        layer(x)


@pytest.mark.parametrize("T", [1, 70])
def test_an_output_of_another_width(T):
    """An output projection that widens is not the layer the one call is made for; the modules take it."""
    layer = _layer(512, 4)
    layer.o_proj = torch.nn.Linear(512, 96, bias=False, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(2, T, 512, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        (o, _, _), labels = _labels(lambda: layer(x))
        want = copy.deepcopy(layer).float()(x.float())[0]
    assert o.shape == (2, T, 96) and "lowrank_gate_fwd" not in labels and rel_l2(o, want) <= 2e-2


def test_in_place_operations_on_the_output():
    """`o += residual`, in-place dropout or activation on a training step's output, as on a linear layer's."""
    layer = _layer(512, 4)
    x = torch.randn(2, 70, 512, device="cuda", dtype=torch.bfloat16)
    grads = []
    for inplace in (False, True):
        leaf = x.clone().requires_grad_()
        o = layer(leaf)[0]
        assert o.grad_fn is not None and not o._is_view()
        if inplace:
            o += leaf
            o.relu_()
        else:
            o = torch.relu(o + leaf)
        grads.append(torch.autograd.grad(o, [leaf, *layer.parameters()], torch.ones_like(o)))
    for a, b in zip(*grads):
        assert torch.equal(a, b)

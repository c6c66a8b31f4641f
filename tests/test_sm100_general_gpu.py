"""The general form of the tcgen05 GLA kernels against the CPU oracle: sequences that do not fill their last chunk,
packed batches (also with sequences cut into runs), K < 128, V beyond one 128-wide slice, constant and absent gates."""
import pytest
import torch

from oracle import gla as O
from oracle import simple_gla as OS
from tests.util import assert_close

pytestmark = pytest.mark.gpu

CASES = [
    # B, T, H, K, V, cu_seqlens
    (1, 65, 1, 128, 128, None),               # one token into the second chunk
    (2, 100, 3, 128, 128, None),
    (3, 127, 16, 128, 128, None),             # 48 blocks: the fused forward
    (1, 1000, 2, 128, 128, None),             # runs of a cut sequence, the last chunk short
    (1, 64 * 11, 2, 128, 128, None),          # whole chunks, a prime number of them
    (2, 130, 2, 64, 128, None),
    (2, 128, 2, 64, 64, None),
    (1, 70, 2, 32, 40, None),                 # the smallest K; V not a multiple of 16
    (1, 200, 2, 128, 256, None),              # two value slices
    (1, 96, 1, 72, 328, None),                # three, the last 72 wide
    (1, 256, 2, 128, 128, [0, 1, 64, 65, 200, 256]),
    (1, 1500, 2, 128, 128, [0, 1200, 1229, 1500]),      # one sequence cut, two whole
    (1, 300, 25, 64, 192, [0, 37, 300]),      # fused, packed, two slices
]


def _inputs(seed, B, T, H, K, V, N, scalar):
    from tops_b200.synth import make_inputs
    x = make_inputs(seed, B, T, H, K, V, dtype=torch.bfloat16, gate="scalar" if scalar else "per_channel", with_grads=True)
    g = torch.Generator().manual_seed(seed)
    x["h0"] = 0.1 * torch.randn(N, H, K, V, generator=g)
    x["dht"] = 0.1 * torch.randn(N, H, K, V, generator=g)
    return x


def _compare(run, x, names, want):
    from tops_b200 import _lib as L
    c = {n: v.cuda() for n, v in x.items()}
    for n in names:
        c[n].requires_grad_()
    L.lib.tops_b200_profile_enable(1)
    o, ht = run(c)
    got = (o, ht, *torch.autograd.grad([o, ht], [c[n] for n in names], [c["do"], c["dht"]]))
    torch.cuda.synchronize()
    L.lib.tops_b200_profile_enable(0)
    import ctypes
    buf = ctypes.create_string_buffer(4096)
    L.lib.tops_b200_profile_read(buf, len(buf))
    assert L.device_error() == 0
    labels = [ln.split()[0] for ln in buf.value.decode().splitlines()]
    assert labels and all(n.startswith("sm100") for n in labels), labels
    for n, a, b in zip(("o", "ht", *("d" + n for n in names)), got, want):
        assert_close(n, a, b, torch.bfloat16)


@pytest.mark.parametrize("B,T,H,K,V,cu", CASES)
def test_per_channel_gate(B, T, H, K, V, cu):
    from tops_b200.ops.gla import chunk_gla
    x = _inputs(61, B, T, H, K, V, B if cu is None else len(cu) - 1, False)
    o, ht = O.chunk_gla(x["q"], x["k"], x["v"], x["g"], None, x["h0"], True, cu_seqlens=cu, chunk_size=64)
    dq, dk, dv, dg, dh0 = O.chunk_gla_bwd(x["q"], x["k"], x["v"], x["g"], None, K ** -0.5, x["h0"], None, None, x["do"],
                                          x["dht"], chunk_size=64, cu_seqlens=cu)
    _compare(lambda c: chunk_gla(c["q"], c["k"], c["v"], c["g"], initial_state=c["h0"], output_final_state=True, cu_seqlens=cu),
             x, ("q", "k", "v", "g", "h0"), (o, ht, dq, dk, dv, dg, dh0))


@pytest.mark.parametrize("gate", ["g", "gamma", "none"])
@pytest.mark.parametrize("B,T,H,K,V,cu", [CASES[i] for i in (1, 2, 3, 5, 8, 10, 11)])
def test_scalar_gates(B, T, H, K, V, cu, gate):
    from tops_b200.ops.simple_gla import chunk_simple_gla
    x = _inputs(62, B, T, H, K, V, B if cu is None else len(cu) - 1, True)
    gamma = -torch.linspace(0.01, 0.2, H) if gate == "gamma" else None
    g = x["g"] if gate == "g" else None
    o, ht = OS.chunk_simple_gla(x["q"], x["k"], x["v"], g, gamma, None, x["h0"], True, cu_seqlens=cu, chunk_size=64)
    dq, dk, dv, dg, dh0 = OS.chunk_simple_gla_bwd(x["q"], x["k"], x["v"], g, gamma, x["h0"], x["do"], x["dht"], K ** -0.5,
                                                  chunk_size=64, cu_seqlens=cu)
    names = ("q", "k", "v", "g", "h0") if gate == "g" else ("q", "k", "v", "h0")
    want = (o, ht, dq, dk, dv, dg, dh0) if gate == "g" else (o, ht, dq, dk, dv, dh0)
    gam = None if gamma is None else gamma.cuda()
    _compare(lambda c: chunk_simple_gla(c["q"], c["k"], c["v"], c["g"] if gate == "g" else None, gam, None, c["h0"], True,
                                        cu_seqlens=cu), x, names, want)


def test_an_infinity_in_one_packed_sequence_stays_there():
    """The short last chunk of a sequence reads on into the next one; nothing of it may get in."""
    from tops_b200.ops.gla import chunk_gla
    cu = [0, 70, 140]
    x = _inputs(63, 1, 140, 2, 128, 128, 2, False)
    clean = {n: v.cuda() for n, v in x.items()}
    dirty = {n: v.clone() for n, v in clean.items()}
    for n in ("q", "k", "v", "g", "do"):
        dirty[n][:, 70:] = float("nan")
    outs = []
    for c in (clean, dirty):
        leaves = [c[n].requires_grad_() for n in ("q", "k", "v", "g")]
        o, ht = chunk_gla(c["q"], c["k"], c["v"], c["g"], output_final_state=True, cu_seqlens=cu)
        grads = torch.autograd.grad([o, ht], leaves, [c["do"], c["dht"]])
        outs.append([o[:, :70], ht[0], *(t[:, :70] for t in grads)])
    for a, b in zip(*outs):
        assert torch.isfinite(b.float()).all() and torch.equal(a, b)


def test_many_short_packed_sequences():
    """More sequences than fit the small table launch."""
    from tops_b200.ops.gla import chunk_gla
    cu = list(range(0, 901, 3))
    x = _inputs(64, 1, 900, 1, 32, 32, 300, False)
    o, ht = O.chunk_gla(x["q"], x["k"], x["v"], x["g"], None, x["h0"], True, cu_seqlens=cu, chunk_size=64)
    dq, dk, dv, dg, dh0 = O.chunk_gla_bwd(x["q"], x["k"], x["v"], x["g"], None, 32 ** -0.5, x["h0"], None, None, x["do"],
                                          x["dht"], chunk_size=64, cu_seqlens=cu)
    _compare(lambda c: chunk_gla(c["q"], c["k"], c["v"], c["g"], initial_state=c["h0"], output_final_state=True, cu_seqlens=cu),
             x, ("q", "k", "v", "g", "h0"), (o, ht, dq, dk, dv, dg, dh0))

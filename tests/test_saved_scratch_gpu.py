"""The scratch a C caller keeps from a chunked forward for its backward: nothing is stored beyond the size it states, and a
scratch that is too small for the kernels that serve the problem is left alone (the backward computes it again)."""
import ctypes as C

import pytest
import torch

from tops_b200.synth import make_inputs

pytestmark = pytest.mark.gpu
BAND = 4096


def _step(x, chunk, elems, stated, cu=None):
    """One forward + backward through the ABI with a scratch of `elems` elements of the input type between guard bands."""
    from tops_b200 import _lib as L
    q, k, v, g, do = (x[n] for n in ("q", "k", "v", "g", "do"))
    (B, T, H, K), V, dev = q.shape, v.shape[-1], q.device
    pb = L.ChunkProblem(B, T, H, K, V, chunk, L.dtype_code(q.dtype), L.dtype_code(g.dtype), L.GATE_PER_CHANNEL, L.IMPL_AUTO, K ** -0.5)
    if stated == "enough":
        stated = L.lib.tops_b200_chunk_saved_bytes(C.byref(pb))
        elems = stated // q.element_size()
    n = elems * q.element_size()
    raw = torch.full((2 * BAND + n,), 0x5A, dtype=torch.uint8, device=dev)
    saved = raw.data_ptr() + BAND if n else None
    st = L.stream_ptr(dev)
    p = L.ChunkFwdParams()
    o = torch.empty_like(v)
    p.pb, p.q, p.k, p.v, p.g, p.o = pb, L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(g), L.ptr(o)
    p.saved_out, p.saved_bytes = saved, stated
    ws = L.workspace(L.lib.tops_b200_chunk_fwd_workspace_bytes(C.byref(p)), dev)
    L.check(L.lib.tops_b200_chunk_gla_fwd(C.byref(p), ws.data_ptr(), ws.numel(), st), "fwd")
    b = L.ChunkBwdParams()
    grads = [torch.empty_like(t, dtype=torch.float32) for t in (q, k, g)] + [torch.empty_like(v)]
    b.pb, b.q, b.k, b.v, b.g, b.do_ = pb, L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(g), L.ptr(do)
    b.dq, b.dk, b.dg, b.dv = (L.ptr(t) for t in grads)
    b.grad_dtype = b.dg_dtype = L.F32
    b.h_saved, b.saved_bytes = saved, stated
    ws = L.workspace(L.lib.tops_b200_chunk_bwd_workspace_bytes(C.byref(b)), dev)
    L.check(L.lib.tops_b200_chunk_gla_bwd(C.byref(b), ws.data_ptr(), ws.numel(), st), "bwd")
    torch.cuda.synchronize()
    assert bool((raw[:BAND] == 0x5A).all()) and bool((raw[BAND + n:] == 0x5A).all())
    return [o, *grads], bool((raw[BAND:BAND + n] != 0x5A).any())


@pytest.mark.parametrize("dtype,chunk,B,T,H,K,V", [(torch.bfloat16, 64, 2, 128, 2, 64, 64), (torch.bfloat16, 64, 1, 100, 2, 64, 128),
                                                   (torch.bfloat16, 64, 1, 64, 2, 128, 192), (torch.bfloat16, 64, 1, 100, 2, 128, 128),
                                                   (torch.bfloat16, 64, 1, 128, 2, 128, 128), (torch.float32, 16, 1, 100, 2, 64, 64)])
def test_scratch_of_a_stated_size(dtype, chunk, B, T, H, K, V):
    x = {n: t.cuda() for n, t in make_inputs(5, B, T, H, K, V, dtype=dtype, with_grads=True).items()}
    elems = B * -(-T // chunk) * H * K * V
    none, _ = _step(x, chunk, 0, 0)
    full, used = _step(x, chunk, 0, "enough")
    assert used
    plain = dtype == torch.bfloat16 and K == V == 128 and T % 64 == 0
    # states, no size, a size that is too small, and one element less than what is needed
    for stated, n in ((0, elems), (elems * x["q"].element_size(), elems), (2, 1)):
        got, used = _step(x, chunk, n if stated != 2 else elems, stated)
        fits = plain and stated != 2   # (the plain form's tiles are what [B,NT,H,K,V] holds)
        if dtype == torch.bfloat16 and V == 128 == K and stated not in (0, 2):
            fits = True                # (so are those of a short last chunk)
        assert used == fits
        for a, b in zip(got, full if fits else none):
            assert torch.equal(a, b)
    for a, b in zip(full, none):       # a kept state is the one that would be computed again, up to its rounding to bf16
        assert ((a.double() - b.double()).norm() / b.double().norm()).item() <= (2e-3 if dtype == torch.bfloat16 else 0)

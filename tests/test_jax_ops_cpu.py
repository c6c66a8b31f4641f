"""The sizes tops_b200/jax_ops.py hands to XLA, with stand-ins for jax and the shim (neither is installed everywhere the
package is): the residual buffer of the chunked forward holds what the C ABI says its kernels keep."""
import ctypes
import importlib.util
import math
import os
import sys
import types

import numpy as np
import pytest

from tops_b200 import _lib as L

PATH = os.path.join(os.path.dirname(L.__file__), "jax_ops.py")


class Struct:
    def __init__(self, shape, dtype):
        self.shape, self.dtype = tuple(shape), np.dtype(dtype)


class Shim:
    def __getattr__(self, name):
        return name


@pytest.fixture
def jax_ops(monkeypatch):
    calls = []

    def ffi_call(name, out, **kw):
        def run(*args, **attrs):
            calls.append((name, out))
            return out
        return run
    jax, jnp, ffi = (types.ModuleType(n) for n in ("jax", "jax.numpy", "jax.ffi"))
    ffi.ffi_call, ffi.pycapsule, ffi.register_ffi_target = ffi_call, lambda f: f, lambda *a, **k: None

    class custom_vjp:
        def __init__(self, fn, nondiff_argnums=()):
            self.fn = fn

        def __call__(self, *args):
            return self.fn(*args)

        def defvjp(self, fwd, bwd):
            self.fwd, self.bwd = fwd, bwd
    jax.ffi, jax.numpy, jax.custom_vjp, jax.ShapeDtypeStruct = ffi, jnp, custom_vjp, Struct
    jnp.float32, jnp.uint8, jnp.dtype = np.float32, np.uint8, np.dtype
    jnp.zeros = lambda shape, dtype: Struct(shape, dtype)
    for m in (jax, jnp, ffi):
        monkeypatch.setitem(sys.modules, m.__name__, m)
    cdll, exists = ctypes.CDLL, os.path.exists
    monkeypatch.setattr(ctypes, "CDLL", lambda p, **kw: Shim() if p.endswith("_jax.so") else cdll(p, **kw))
    monkeypatch.setattr(os.path, "exists", lambda p: p.endswith("_jax.so") or exists(p))
    spec = importlib.util.spec_from_file_location("jax_ops_under_test", PATH)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod, calls


@pytest.mark.parametrize("B,T,H,K,V,chunk,scalar", [(2, 100, 3, 64, 64, 16, False), (1, 64, 2, 64, 128, 64, False), (1, 65, 1, 16, 256, 32, True),
                                                    (1, 50, 2, 128, 128, 16, False)])
def test_residual_buffer_holds_what_the_abi_keeps(jax_ops, B, T, H, K, V, chunk, scalar):
    mod, calls = jax_ops
    q, v = Struct((B, T, H, K), np.float32), Struct((B, T, H, V), np.float32)
    g = Struct((B, T, H) if scalar else q.shape, np.float32)
    mod.chunk_gla(q, q, v, g, chunk_size=chunk)
    (name, out), = calls
    pb = L.ChunkProblem(B, T, H, K, V, chunk, L.F32, L.F32, L.GATE_SCALAR if scalar else L.GATE_PER_CHANNEL, L.IMPL_AUTO, K ** -0.5)
    want = L.lib.tops_b200_chunk_saved_bytes(ctypes.byref(pb))
    saved = out[2]
    assert name == "tops_b200_ffi_chunk_fwd" and math.prod(saved.shape) * saved.dtype.itemsize == want

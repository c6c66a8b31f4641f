"""The fp32 CUDA-core backward on the states its forward kept against the one that computes them again."""
import pytest
import torch

from tops_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,V,cu", [(64, 64, None), (64, 64, [0, 1, 40, 200]), (40, 24, None), (72, 64, None)])
def test_fp32_backward_on_kept_states(K, V, cu):
    from tops_b200.ops.gla import chunk_gla, chunk_gla_bwd
    T, H, N = 200, 3, 1 if cu is None else len(cu) - 1
    x = make_inputs(83, 1, T, H, K, V, dtype=torch.float32, with_grads=True)
    gen = torch.Generator().manual_seed(83)
    x["h0"], x["dht"] = torch.randn(N, H, K, V, generator=gen), torch.randn(N, H, K, V, generator=gen)
    c = {n: t.cuda() for n, t in x.items()}
    again = chunk_gla_bwd(c["q"], c["k"], c["v"], c["g"], None, K ** -0.5, c["h0"], None, None, c["do"], c["dht"], chunk_size=16,
                          cu_seqlens=cu)
    leaves = [c[n].requires_grad_() for n in ("q", "k", "v", "g", "h0")]
    o, ht = chunk_gla(c["q"], c["k"], c["v"], c["g"], initial_state=c["h0"], output_final_state=True, cu_seqlens=cu, chunk_size=16)
    kept = torch.autograd.grad([o, ht], leaves, [c["do"], c["dht"]])
    for a, b in zip(kept, again):
        assert torch.equal(a, b)

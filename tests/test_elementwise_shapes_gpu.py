"""The gate and norm kernels at the sizes where their thread layouts change: vectors of four and of eight elements, rows
shared by 1 to 32 lanes, several vectors per lane, one row, more columns than a block has threads."""
import pytest
import torch

from oracle import aux as O
from tests.util import assert_close

pytestmark = pytest.mark.gpu


def _grads(fn, inputs, dy):
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    y = fn(*leaves)
    return [y.detach(), *torch.autograd.grad(y, leaves, dy.to(y.dtype))]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(1, 4), (3, 8), (65, 12), (7, 72), (33, 136), (5, 260), (9, 516), (2, 1000), (31, 1024)])
def test_row_kernels(dtype, rows, D):
    from tops_b200.ops.norm import l2norm, rmsnorm_gated
    gen = torch.Generator().manual_seed(rows * D)
    x, g, dy = (torch.randn(rows, D, generator=gen).to(dtype) for _ in range(3))
    w = 1 + 0.1 * torch.randn(D, generator=gen)
    for f, ref, args in ((l2norm, O.l2norm, (x,)), (rmsnorm_gated, O.rmsnorm_gated, (x, g, w))):
        want = _grads(ref, args, dy)
        got = _grads(f, [t.cuda() for t in args], dy.cuda())
        for i, (a, b) in enumerate(zip(got, want)):
            assert_close(f"{f.__name__} {i}", a.float().cpu(), b.float(), dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lower_bound", [None, -5.0])
@pytest.mark.parametrize("rows,H,K", [(1, 1, 4), (5, 3, 12), (700, 2, 40), (3, 5, 512), (1300, 1, 8)])
def test_gate_kernels(dtype, lower_bound, rows, H, K):
    from tops_b200.ops.gate import gla_gate, kda_gate_fwd
    gen = torch.Generator().manual_seed(rows + H * K)
    # (up to +-20: both tails of the softplus)
    g = (8 * torch.randn(rows, H, K, generator=gen)).clamp(-20, 20).to(dtype)
    dy = torch.randn(rows, H, K, generator=gen)
    A, bias = 0.5 * torch.randn(H, generator=gen), torch.randn(H * K, generator=gen)
    want = _grads(lambda a, b, c: O.kda_gate_fwd(a, b, c, lower_bound), (g, A, bias), dy)
    got = _grads(lambda a, b, c: kda_gate_fwd(a, b, c, lower_bound), (g.cuda(), A.cuda(), bias.cuda()), dy.cuda())
    assert_close("y", got[0].cpu(), want[0], torch.float32)
    assert_close("dg", got[1].float().cpu(), want[1].float(), dtype)
    for name, a, r in (("dA_log", got[2], want[2]), ("dbias", got[3], want[3])):   # sums over rows: relative bar
        assert ((a.cpu() - r).norm() / r.norm()).item() <= (1e-4 if dtype == torch.float32 else 1e-2), name
    if lower_bound is None:
        want = _grads(lambda a: O.gla_gate(a, 16.0, None), (g,), dy)
        got = _grads(lambda a: gla_gate(a, 16.0, None), (g.cuda(),), dy.cuda())
        for a, b in zip(got, want):
            assert_close("gla_gate", a.float().cpu(), b.float(), dtype)


@pytest.mark.parametrize("shape", [(2, 3, 0), (0, 3, 64), (2, 0, 64)])
def test_tensors_without_elements_are_refused(shape):
    """Rows of no channels, no rows, no heads: an error that can be caught, in whatever layer finds it."""
    from tops_b200._lib import TopsError
    from tops_b200.ops.gate import gla_gate, kda_gate_fwd
    from tops_b200.ops.norm import l2norm, rmsnorm_gated
    x = torch.empty(shape, device="cuda", dtype=torch.bfloat16)
    for call in (lambda: l2norm(x), lambda: rmsnorm_gated(x, x), lambda: gla_gate(x), lambda: kda_gate_fwd(x, torch.zeros(3, device="cuda"))):
        with pytest.raises((AssertionError, TopsError)):
            call()


def test_fp32_results_keep_fp32_precision():
    """Against fp64, fp32 tensors.  The bars are what CUDA's division and log1pf leave on these inputs (results, gradients),
    plus 1 %; the approximate reciprocal and the polynomial of the 16-bit kernels leave 1 - 5 % more."""
    from tops_b200.ops.gate import gla_gate, kda_gate_fwd
    from tops_b200.ops.norm import l2norm, rmsnorm_gated
    gen = torch.Generator(device="cuda").manual_seed(5)
    x, z, dy = (torch.randn(2, 1500, 8, 128, generator=gen, device="cuda") for _ in range(3))
    A = torch.randn(8, generator=gen, device="cuda")
    F = torch.nn.functional
    e = A.double().exp()[:, None]
    cases = [(lambda t: kda_gate_fwd(t, A, lower_bound=-5.0), lambda t: -5 * torch.sigmoid(e * t), 5.092e-8, 1.128e-7),
             (lambda t: gla_gate(t), lambda t: F.logsigmoid(t) / 16, 3.208e-8, 5.525e-8),
             (lambda t: kda_gate_fwd(t, A), lambda t: -e * F.softplus(t), 5.817e-8, 6.566e-8),
             (lambda t: l2norm(t), lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6), 4.677e-8, 5.377e-8),
             (lambda t: rmsnorm_gated(t, z), lambda t: t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-5) * F.silu(z.double()),
              7.186e-8, 7.729e-8)]
    for op, ref, *bars in cases:
        leaf, exact = x.clone().requires_grad_(), x.double().requires_grad_()
        y, want = op(leaf), ref(exact)
        pairs = [(y, want), (torch.autograd.grad(y, leaf, dy)[0], torch.autograd.grad(want, exact, dy.double())[0])]
        for (a, b), bar in zip(pairs, bars):
            err = ((a.double() - b).norm() / b.norm()).item()
            assert err <= 1.01 * bar, (err, bar)

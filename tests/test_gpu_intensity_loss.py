"""The loss of a phase-only hologram as kernels (csrc/epilogue.cu) against its definition in
array operations.

Both form the same sums in FP64 in another order, each of at most 70001 terms through trees and
short chains: 1e-13 of the largest value is far above their rounding and far below any mistake."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

TOL = 1e-13


def _ops():
    import __graft_entry__ as g
    g.load_package()
    from holo_gb300 import torch_ops
    return torch_ops


def _case(m, seed=0):
    gen = torch.Generator().manual_seed(seed)
    z = torch.randn(m, 2, generator=gen, dtype=torch.float64) * 3
    t = torch.rand(m, generator=gen, dtype=torch.float64)
    return z.cuda(), t.cuda()


def _near(a, b):
    a, b = a.detach(), b.detach()
    return bool((a - b).abs().max() <= TOL * b.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 2, 255, 1024, 1025, 4097, 70001, 600001])
def test_loss_and_gradient(m):
    ops = _ops()
    z, t = _case(m, m)
    a, b = z.clone().requires_grad_(True), z.clone().requires_grad_(True)
    la, lb = ops.intensity_loss(a, t), ops._intensity_loss_ops(b, t)
    assert la.shape == lb.shape and la.dtype == lb.dtype
    assert type(la.grad_fn).__name__ == "_IntensityLossBackward"
    (3.0 * la).backward()
    (3.0 * lb).backward()
    assert _near(la, lb) and _near(ops.intensity_loss(z, t), lb)
    # m = 1: I / mean I is 1 whatever z is, both gradients are rounding
    assert _near(a.grad, b.grad) if m > 1 else float(a.grad.abs().max()) < TOL


@pytest.mark.gpu
def test_what_the_array_operations_allow():
    """Second derivatives, batched gradients, a target that changes before the gradient, a
    modified field refused, infinities and NaN, transforms and forward mode."""
    ops = _ops()
    z, t = _case(2000)
    a, b = z.clone().requires_grad_(True), z.clone().requires_grad_(True)
    w = torch.randn_like(z)
    hv = []
    for x, f in ((a, ops.intensity_loss), (b, ops._intensity_loss_ops)):
        g, = torch.autograd.grad(f(x, t), x, create_graph=True)
        hv.append(torch.autograd.grad((g * w).sum(), x)[0])
    assert _near(hv[0], hv[1])
    many = torch.arange(1.0, 4.0, dtype=torch.float64, device="cuda")
    ga, = torch.autograd.grad(ops.intensity_loss(a, t), a, many, is_grads_batched=True)
    gb, = torch.autograd.grad(ops._intensity_loss_ops(b, t), b, many, is_grads_batched=True)
    assert _near(ga, gb)
    moving = t.clone()
    la = ops.intensity_loss(a, moving)
    moving.zero_()
    assert _near(torch.autograd.grad(la, a)[0], gb[0])
    x = z.clone().requires_grad_(True)
    y = x * 1.0
    la = ops.intensity_loss(y, t)
    y.mul_(2.0)
    with pytest.raises(RuntimeError):
        la.backward()
    for value in (float("inf"), float("nan"), 0.0):
        bad = z.clone() if value else torch.zeros_like(z)
        bad[5, 0] = value
        assert np.array_equal(ops.intensity_loss(bad, t).cpu(), ops._intensity_loss_ops(bad, t).cpu(),
                              equal_nan=True)
    gf = torch.func.grad(lambda q: ops.intensity_loss(q, t))(z)
    assert _near(gf, gb[0])
    many_z = torch.stack([z, 2 * z, -z])
    assert _near(torch.func.vmap(lambda q: ops.intensity_loss(q, t))(many_z),
                 torch.stack([ops._intensity_loss_ops(q, t) for q in many_z]))
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(z, w)
        tangent = torch.autograd.forward_ad.unpack_dual(ops.intensity_loss(d, t)).tangent
    assert _near(tangent, (gb[0] * w).sum())


@pytest.mark.gpu
def test_forms_that_stay_array_operations():
    """Other types, strides, offsets, shapes and devices give what they gave."""
    ops = _ops()
    z, t = _case(512)
    wide = torch.randn(512, 3, dtype=torch.float64, device="cuda")
    odd = torch.cat([z.reshape(-1)[:1], z.reshape(-1)])[1:].reshape(512, 2)  # 8 bytes off
    forms = [(z.float(), t), (z, t.float()), (z.t().contiguous().t(), t), (odd, t),
             (wide[:, 1:], t), (wide, t), (z[::2], t[::2]), (z, t[:1]), (z.cpu(), t.cpu()),
             (z, t.clone().requires_grad_(True)), (torch._neg_view(z), t), (z, torch._neg_view(t))]
    for a, b in forms:
        want = ops._intensity_loss_ops(a, b)
        got = ops.intensity_loss(a, b)
        assert got.dtype == want.dtype and got.device == want.device
        assert torch.equal(got, want)
    for a, b in ((z, t[:7]), (z[:, 0], t)):
        with pytest.raises((RuntimeError, IndexError)):
            ops.intensity_loss(a, b)


@pytest.mark.gpu
def test_capture_and_a_second_stream():
    ops = _ops()
    z, t = _case(3000)
    z.requires_grad_(True)
    want = torch.autograd.grad(ops.intensity_loss(z, t), z)[0]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            got = torch.autograd.grad(ops.intensity_loss(z, t), z)[0]
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(got, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = torch.autograd.grad(ops.intensity_loss(z, t), z)[0]
    got.zero_()
    graph.replay()
    assert torch.equal(got, want)

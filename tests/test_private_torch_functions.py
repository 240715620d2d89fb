"""The loss and the call path do without those private PyTorch functions that a version may lack."""
import pytest

PRIVATE = ["_are_functorch_transforms_active", "_len_torch_dispatch_stack",
           "_len_torch_function_stack", "_has_storage"]


def _loss(holo, device, monkeypatch, name):
    import torch
    from holo_gb300 import torch_ops
    g = torch.Generator().manual_seed(0)
    z = torch.rand(50, 2, generator=g, dtype=torch.float64).to(device).requires_grad_(True)
    target = torch.rand(50, generator=g, dtype=torch.float64).to(device)
    with monkeypatch.context() as m:  # PyTorch's own backward asks for some of them
        m.delattr(torch._C, name)
        loss = torch_ops.intensity_loss(z, target)
    loss.backward()
    inten = (z.detach() ** 2).sum(1)
    want = torch.mean((inten / inten.mean() - target) ** 2)
    assert abs(loss.item() - want.item()) < 1e-12 and torch.isfinite(z.grad).all()


@pytest.mark.parametrize("name", PRIVATE)
def test_loss_without(holo, monkeypatch, name):
    _loss(holo, "cpu", monkeypatch, name)


@pytest.mark.gpu
@pytest.mark.parametrize("name", PRIVATE + ["_cuda_getCurrentRawStream"])
def test_on_the_gpu_without(holo, monkeypatch, name):
    import torch
    if name == "_cuda_getCurrentRawStream":
        x = torch.rand(2000, dtype=torch.float64, device="cuda:0")
        monkeypatch.delattr(torch._C, name)
        amp, phase, _ = holo.normalize_polar(x)
        assert amp.max().item() <= 1 and phase.isfinite().all()
    else:
        _loss(holo, "cuda:0", monkeypatch, name)

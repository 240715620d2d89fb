"""NaN and infinite values in sums by cluster expansions: a source whose amplitude, phase or position
is not finite leaves no target with a finite value, as the pair-by-pair sum has it; a target whose
position is not finite spoils its own value only."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2

pytestmark = pytest.mark.gpu

N, M = 16384, 262144
BAD = ["amp_nan", "amp_inf", "amp_huge", "phase_nan", "phase_inf", "source_nan", "source_flat_nan"]


def _t(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")


def _set():
    rng = np.random.default_rng(5)
    u, v = grid(128, 10e-6, 0.3), grid(512, 7.56e-6, 0.0)
    return rng.uniform(0, 1, N), rng.uniform(0, 2 * np.pi, N), u, v


def _spoil(kind, at, amp, phase, u):
    if kind == "amp_nan":
        amp[at] = np.nan
    elif kind == "amp_inf":
        amp[at] = -np.inf
    elif kind == "amp_huge":
        amp[at] = 1e200  # an infinity in FP32
    elif kind == "phase_nan":
        phase[at] = np.nan
    elif kind == "phase_inf":
        phase[at] = np.inf
    elif kind == "source_nan":
        u[at, 0] = np.nan
    else:
        u[at, 2] = np.nan  # along the axis that the clusters' nodes leave out


def _execute(holo, amp, phase, u, v, sign=-1):
    with holo.Plan(_t(u), _t(v), "split32") as plan:
        n0 = holo.api.kernel_launches()
        y = plan.execute(_t(amp), _t(phase), sign, LAM)
        assert holo.api.kernel_launches() - n0 in (5, 6)  # by expansions
    return y.cpu().numpy()


@pytest.mark.parametrize("at", [0, 8191, N - 1])
@pytest.mark.parametrize("kind", BAD)
def test_no_target_stays_finite(holo, kind, at):
    amp, phase, u, v = _set()
    _spoil(kind, at, amp, phase, u)
    y = _execute(holo, amp, phase, u, v)
    assert not np.any(np.isfinite(y.real) & np.isfinite(y.imag))


def test_a_bad_target_is_alone(holo):
    amp, phase, u, v = _set()
    v[777] = np.nan
    y = _execute(holo, amp, phase, u, v)
    bad = ~(np.isfinite(y.real) & np.isfinite(y.imag))
    assert bad[777] and bad.sum() == 1
    idx = np.arange(700, M, 513)
    assert rel_l2(y[idx], holo.transform(amp, phase, u, v[idx], -1, LAM, precision="fp64")) < 2.5e-6


def test_batch(holo):
    import torch
    amp, phase, u, v = _set()
    y = [torch.zeros(2 * M, dtype=torch.float64, device="cuda:0") for _ in range(3)]
    bad = amp.copy()
    bad[12345] = np.nan
    problems = [holo.Problem(_t(a), _t(phase), _t(u), _t(v), -1, LAM, y[i])
                for i, a in enumerate((amp, bad, amp))]
    with holo.Batch(problems) as batch:
        batch.execute()
    torch.cuda.synchronize()
    assert torch.isfinite(y[0]).all() and torch.isfinite(y[2]).all()
    assert not torch.isfinite(y[1].view(-1, 2)).all(1).any()


def test_a_nan_loss_gives_a_nan_gradient(holo):
    import torch
    from holo_gb300 import torch_ops
    amp, phase, u, v = _set()
    target = torch.ones(M, dtype=torch.float64, device="cuda:0")
    target[99] = float("nan")
    with holo.Plan(_t(u), _t(v), "split32") as plan:
        ph = _t(phase).requires_grad_(True)
        loss = torch_ops.intensity_loss(torch_ops.huygens(_t(amp), ph, plan, 1, LAM), target)
        loss.backward()
    assert torch.isnan(loss).item() and not torch.isfinite(ph.grad).any()

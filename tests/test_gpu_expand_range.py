"""Sums by cluster expansions whose amplitudes are all faint or all bright: the same relative error
whatever the amplitudes' common factor (FP32 numbers down to 1.2e-38 keep 24 bits)."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2

pytestmark = pytest.mark.gpu

TOL = 2.5e-6  # of the field, as for amplitudes near 1


@pytest.mark.parametrize("factor", [1e-36, 3e-34, 1e-30, 1e-12, 1e12, 1e30, 3e37])
@pytest.mark.parametrize("batched", [False, True])
def test_common_factor(holo, factor, batched):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")
    rng = np.random.default_rng(6)
    u, v = grid(128, 10e-6, 0.3), grid(400, 7.56e-6, 0.0)
    amp, phase = rng.uniform(0.1, 1, len(u)), rng.uniform(0, 2 * np.pi, len(u))
    idx = np.arange(0, len(v), 101)
    want = holo.transform(amp, phase, u, v[idx], 1, LAM, precision="fp64")
    if batched:
        y = torch.zeros(2 * len(v), dtype=torch.float64, device="cuda:0")
        with holo.Batch([holo.Problem(t(amp * factor), t(phase), t(u), t(v), 1, LAM, y)]) as batch:
            batch.execute()
        y = torch.view_as_complex(y.view(-1, 2))
    else:
        with holo.Plan(t(u), t(v), "split32") as plan:
            n0 = holo.api.kernel_launches()
            y = plan.execute(t(amp * factor), t(phase), 1, LAM)
            assert holo.api.kernel_launches() - n0 in (5, 6)
    assert rel_l2(y.cpu().numpy()[idx] / factor, want) < TOL

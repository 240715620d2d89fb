"""The split path's stated accuracy, 1e-5 of the field (include/holo.h), at the sizes on both sides
of the rules that choose its kernels; plans, one-shot calls and batches."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("n,m,z", [
    (30000, 3000, 0.35), (3000, 30000, 0.35), (65536, 4096, 0.35), (256, 65537, 0.35),
    (1024, 100000, 0.3), (12345, 999, 0.1), (5000, 5000, 0.02), (256, 512, 0.4), (257, 512, 0.4),
    (1025, 4097, 0.4), (300, 38913, 0.4), (76 * 1024 + 1, 512, 0.4)])
def test_within_1e_5(holo, n, m, z):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")
    rng = np.random.default_rng(n + m)
    u = grid(int(np.ceil(np.sqrt(n))), 10e-6, z)[:n]
    v = grid(int(np.ceil(np.sqrt(m))), 7.56e-6, 0.0)[:m]
    u[:, :2] += rng.uniform(-2e-6, 2e-6, (n, 2))
    u = u[rng.permutation(n)]
    amp, phase = rng.uniform(0, 1, n), rng.uniform(0, 2 * np.pi, n)
    want = holo.transform(amp, phase, u, v, -1, LAM, precision="fp64")
    assert rel_l2(holo.transform(amp, phase, u, v, -1, LAM), want) < TOL
    with holo.Plan(u, v) as plan:
        assert rel_l2(plan.execute(amp, phase, -1, LAM), want) < TOL
    y = torch.zeros(2 * m, dtype=torch.float64, device="cuda:0")
    with holo.Batch([holo.Problem(t(amp), t(phase), t(u), t(v), -1, LAM, y)]) as batch:
        batch.execute()
    assert rel_l2(torch.view_as_complex(y.view(-1, 2)).cpu().numpy(), want) < TOL

"""Calls that plan for one use: sizes on both sides of the rules that choose between packed and
Hilbert tiles and between the pair kernel and cluster expansions, against FP64 sums.

2e-5 of the field is what the split path is held to."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [-1, 1])
@pytest.mark.parametrize("n,m,z", [
    (30000, 3000, 0.35), (3000, 30000, 0.35), (65536, 4096, 0.35), (256, 65537, 0.35),
    (1024, 100000, 0.3), (12345, 999, 0.1), (5000, 5000, 0.02)])
def test_one_shot(holo, n, m, z, sign):
    rng = np.random.default_rng(n + m)
    u = grid(int(np.ceil(np.sqrt(n))), 10e-6, z)[:n]
    v = grid(int(np.ceil(np.sqrt(m))), 7.56e-6, 0.0)[:m]
    u[:, :2] += rng.uniform(-2e-6, 2e-6, (n, 2))
    shuffle = rng.permutation(n)
    u = u[shuffle]
    amp, phase = rng.uniform(0, 1, n), rng.uniform(0, 2 * np.pi, n)
    want = holo.transform(amp, phase, u, v, sign, LAM, precision="fp64")
    assert rel_l2(holo.transform(amp, phase, u, v, sign, LAM), want) < 2e-5
    with holo.Plan(u, v) as plan:
        assert rel_l2(plan.execute(amp, phase, sign, LAM), want) < 2e-5

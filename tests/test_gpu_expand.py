"""Sums by cluster expansions (csrc/kernel_expand.cu) against the FP64 kernel.

Tolerance: a field is the product of three factors per point or pair of nodes whose sines and
cosines come from MUFU (absolute error at most 2^-20.5 = 6.7e-7, about 3e-7 rms each), plus
the interpolation (2.5e-7 of the norm) and the TF32 splits (2^-21): 1e-6 rms in all; 2.5e-6
leaves room for the FP32 curvature terms, (h_s + h_t)^2 k / 2r of up to 10 rad.
The sizes end clusters, blocks of 128 targets, groups of 32 source and 64 target clusters
and stages of 64 sources early and late; each set is flat along each axis in turn.
"""
import math

import numpy as np
import pytest

from conftest import LAM, grid, rel_l2

pytestmark = pytest.mark.gpu

TOL = 2.5e-6


def _launches(holo, fn):
    n0 = holo.api.kernel_launches()
    y = fn()
    return y, holo.api.kernel_launches() - n0


def _square(n, pitch, z):
    return grid(math.ceil(math.sqrt(n)), pitch, z)[:n]


# (sources, targets, distance, flat axis, sign, wavelength, lateral offset)
CASES = [
    (16384, 262144, 0.30, 2, -1, LAM, 0.0),
    (16385, 131073, 0.35, 2, 1, LAM, 0.0),       # one point into the next cluster on both sides
    (40063, 100127, 0.41, 2, 1, 650e-9, 0.7e-3),  # ragged, off the axis
    (150001, 40001, 0.50, 1, -1, LAM, 0.0),      # more than 32 source clusters
    (9000, 500001, 0.45, 0, -1, 400e-9, 0.0),    # more than 64 target clusters
    (65536, 65536, 0.20, 2, 1, LAM, 1e-3),       # close: small clusters
    (1000003, 4097, 0.35, 2, 1, LAM, 0.0),       # few targets: split over the source clusters
    (4097, 1000003, 0.35, 1, -1, LAM, 0.0),      # few sources
]


@pytest.mark.parametrize("n,m,dist,flat,sign,lam,dx", CASES)
def test_expansion_against_fp64(holo, n, m, dist, flat, sign, lam, dx):
    import torch
    dev = torch.device("cuda:0")
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device=dev)
    rng = np.random.default_rng(n % 1000 + m % 1000)
    u, v = _square(n, 10e-6, dist), _square(m, 7.56e-6, 0.0)
    u[:, 0] += dx
    u[:, :2] += rng.uniform(-0.5, 0.5, (n, 2)) * 10e-6
    perm = [(a + flat + 1) % 3 for a in range(3)]  # column 2 (the heights) becomes `flat`
    u, v = (np.ascontiguousarray(p[:, np.argsort(perm)]) for p in (u, v))
    assert np.ptp(v[:, flat]) == 0.0 and np.ptp(u[:, flat]) == 0.0
    amp, phase = rng.uniform(0, 1, n), rng.uniform(0, 2 * np.pi, n)
    da, dp = t(amp), t(phase)
    with holo.Plan(t(u), t(v), "split32") as pl:
        y, launches = _launches(holo, lambda: pl.execute(da, dp, sign, lam))
        again = pl.execute(da, dp, sign, lam)
    assert launches in (5, 6), launches  # gather, set-up, moments, translate, targets (, reduce)
    assert torch.equal(y, again)
    idx = np.unique(np.concatenate([np.arange(min(m, 130)), np.arange(max(0, m - 130), m),
                                    rng.choice(m, min(m, 800), replace=False)]))
    y64 = holo.transform(da, dp, t(u), t(v[idx]), sign, lam, precision="fp64").cpu().numpy()
    assert rel_l2(y.cpu().numpy()[idx], y64) < TOL
    holo.handle(0).status()


def test_zero_amplitudes_and_single_cluster_values(holo):
    """Zero amplitudes give a zero field; one bright source among zeros gives its own wave."""
    import torch
    dev = torch.device("cuda:0")
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device=dev)
    u, v = _square(30000, 10e-6, 0.35), _square(150000, 7.56e-6, 0.0)
    amp, phase = np.zeros(len(u)), np.zeros(len(u))
    with holo.Plan(t(u), t(v), "split32") as pl:
        y, launches = _launches(holo, lambda: pl.execute(t(amp), t(phase), 1, LAM))
        assert launches in (5, 6)
        assert torch.count_nonzero(torch.view_as_real(y)).item() == 0
        amp[17123] = 2.0
        y = pl.execute(t(amp), t(phase), 1, LAM).cpu().numpy()
    r = np.linalg.norm(v - u[17123], axis=1)
    assert rel_l2(y, 2.0 * np.exp(1j * 2 * np.pi / LAM * r) / r) < TOL


def test_tilted_and_thick_sets_stay_with_the_pair_kernel(holo):
    """Clusters that are not flat along one common axis have no node grid: the pair kernel."""
    rng = np.random.default_rng(3)
    u, v = _square(20000, 10e-6, 0.35), _square(150000, 7.56e-6, 0.0)
    amp, phase = rng.uniform(0, 1, len(u)), rng.uniform(0, 2 * np.pi, len(u))
    tilt = u.copy()
    tilt[:, 2] += 0.1 * u[:, 0]
    for s in (tilt, u + rng.uniform(-1e-5, 1e-5, u.shape)):
        with holo.Plan(s, v, "split32") as pl:
            y, launches = _launches(holo, lambda: pl.execute(amp, phase, -1, LAM))
        assert launches <= 3, launches
        idx = np.arange(0, len(v), 997)
        assert rel_l2(y[idx], holo.transform(amp, phase, s, v[idx], -1, LAM, precision="fp64")) < 1e-5

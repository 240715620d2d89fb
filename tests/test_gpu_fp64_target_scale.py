"""The fixed-point FP64 kernel (variants 6 and 7) where the targets of one thread lie at very
different distances from a tile's scale source, the brightest of its 64 (the last of equals): every
target against the FP64 pipe's kernel (variant 0), relative to its
own sum of |a| / r.

Each of 64 terms is off by at most 1.5 units, a unit at most 2^-52 of the largest term: 64 x 1.5 x
2^-52 = 2.1e-14 at the very worst, and the errors are as often up as down: 1e-14."""
import numpy as np
import pytest

from conftest import LAM, grid

pytestmark = pytest.mark.gpu

TOL = 1e-14


def _check(holo, amp, phase, u, v, kernel, sign=1):
    x, y = (holo.transform(amp, phase, u, v, sign, LAM, precision="fp64", variant=k)
            for k in (kernel, 0))
    fin = np.isfinite(y.real) & np.isfinite(y.imag)
    assert np.array_equal(fin, np.isfinite(x.real) & np.isfinite(x.imag))
    scale = np.array([np.sum(np.abs(amp) / np.linalg.norm(u - t, axis=1)) for t in v[fin]])
    assert np.max(np.abs(x[fin] - y[fin]) / scale) < TOL


@pytest.mark.parametrize("kernel", [6, 7])
@pytest.mark.parametrize("gap", [1e-18, 1e-15, 1e-12, 1e-9, 1e-7, 1e-5])
@pytest.mark.parametrize("slot", [0, 1, 3])
def test_scale_source_near_a_target(holo, kernel, gap, slot):
    rng = np.random.default_rng(7)
    u, v = grid(8, 10e-6, 0.3), grid(30, 7.56e-6, 0.0)
    for last in (63, 15):  # the last of tiles of 64 and of 16 sources
        s = u.copy()
        s[last] = v[100 + slot] + [0.0, 0.0, gap]
        _check(holo, np.ones(64), rng.uniform(0, 2 * np.pi, 64), s, v, kernel)


@pytest.mark.parametrize("kernel", [6, 7])
@pytest.mark.parametrize("far", [1e-3, 1.0, 1e4])
def test_near_and_far_targets_in_turn(holo, kernel, far):
    rng = np.random.default_rng(8)
    u = grid(20, 10e-6, 0.0)
    v = grid(40, 7.56e-6, 1e-6)
    v[1::2, 2] = far
    v[2::4, 2] = far * 1e-2
    _check(holo, rng.uniform(0.5, 1, 400), rng.uniform(0, 2 * np.pi, 400), u, v, kernel)

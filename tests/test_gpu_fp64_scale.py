"""The fixed-point FP64 kernel (variants 6 and 7) where a tile's scale source, the brightest of its
64 (the last of equals), lies on a target: every target against the FP64 pipe's kernel (variant 0), relative to its
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
@pytest.mark.parametrize("slot", [0, 1, 3])
@pytest.mark.parametrize("last", [63, 15])  # the last of tiles of 64 and of 16 sources
def test_scale_source_on_a_target(holo, kernel, slot, last):
    rng = np.random.default_rng(7)
    u, v = grid(8, 10e-6, 0.3), grid(30, 7.56e-6, 0.0)
    u[last] = v[100 + slot]
    _check(holo, np.ones(64), rng.uniform(0, 2 * np.pi, 64), u, v, kernel)


@pytest.mark.parametrize("kernel", [6, 7])
def test_one_source_on_the_first_target(holo, kernel):
    v = grid(30, 7.56e-6, 0.0)
    _check(holo, np.array([1.5]), np.array([0.3]), v[:1].copy(), v, kernel)


@pytest.mark.parametrize("kernel", [6, 7])
def test_faint_sources_beside_a_bright_one_out_of_range(holo, kernel):
    """Where the scale source's own pair has no fixed-point form, no rounding is made up for it."""
    rng = np.random.default_rng(9)
    u, v = grid(8, 10e-6, 0.3), grid(30, 7.56e-6, 0.0)
    amp = np.full(64, 1e-9)
    amp[63] = 1.0
    u[63] = v[401] + [0.0, 0.0, 1e-16]
    _check(holo, amp, rng.uniform(0, 2 * np.pi, 64), u, v, kernel)

"""Polar form of a field and the adjoint's phase factors (csrc/epilogue.cu, csrc/fp64_fixed.cuh).

The angle is a table angle plus a series of a remainder that is exact to 2^-60, rounded twice: below 3
units in its last place; the modulus is a rounded root of a sum rounded twice: below 1.5.  NumPy's
long double has at least 11 more bits than either."""
import numpy as np
import pytest


def _fields():
    rng = np.random.default_rng(5)
    n = 200000
    angle = rng.uniform(-np.pi, np.pi, n)
    angle[::4] *= 2.0 ** -rng.integers(0, 30, len(angle[::4]))
    angle[1::4] = np.pi / 2 * rng.integers(-2, 3, len(angle[1::4])) + rng.normal(size=len(angle[1::4])) * 1e-6
    radius = 2.0 ** rng.uniform(-60, -21, n)  # below 1e-6: left unnormalised
    return radius * np.exp(1j * angle)


def _ulps(got, want):
    return np.max(np.abs((got - want) / np.spacing(np.abs(want).astype(np.float64)).astype(np.longdouble)))


@pytest.mark.gpu
def test_modulus_and_angle(holo):
    y = _fields()
    amp, phase, top = holo.normalize_polar(y.view(np.float64))
    x, z = y.real.astype(np.longdouble), y.imag.astype(np.longdouble)
    mod = np.sqrt(x * x + z * z)
    assert top == np.float64(mod.max()) or abs(top - mod.max()) <= 2 * np.spacing(top)
    assert _ulps(amp, mod) < 1.5 and _ulps(phase, np.arctan2(z, x)) < 3


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 300001, 700001])
def test_normalised(holo, n):
    rng = np.random.default_rng(n)
    y = rng.normal(size=n) + 1j * rng.normal(size=n)
    amp, phase, top = holo.normalize_polar(y.view(np.float64))
    x, z = y.real.astype(np.longdouble), y.imag.astype(np.longdouble)
    mod = np.sqrt(x * x + z * z)
    assert abs(top - mod.max()) <= 2 * np.spacing(top)
    assert _ulps(amp, mod / mod.max()) < 4  # the maximum's own rounding, the quotient's, the root's
    assert _ulps(phase, np.arctan2(z, x)) < 3


@pytest.mark.gpu
def test_values_without_a_normal_form(holo):
    """Signed zeros, axes, subnormal, huge, infinite and NaN parts: as NumPy's hypot and arctan2,
    with a small and with a normalising maximum."""
    inf, nan, sub = np.inf, np.nan, 5e-324
    parts = [0.0, -0.0, 1e-9, -1e-9, sub, -sub, 1e-300, -3e-160]
    for more in ([], [2.0, -3.0], [1e150, -1e200], [1e300, 1e-300]):
        p = parts + more
        y = np.array([complex(a, b) for a in p for b in p])
        amp, phase, top = holo.normalize_polar(y.view(np.float64))
        want = np.hypot(y.real, y.imag)
        assert abs(top - want.max()) <= 2 * np.spacing(want.max())
        if top >= 1e-6:
            want = np.hypot(y.real / top, y.imag / top)
            angle = np.arctan2(y.imag / top, y.real / top)
        else:
            angle = np.arctan2(y.imag, y.real)
        normal = want > 1e-290
        assert np.all(np.abs(amp - want)[normal] <= 4 * np.spacing(want[normal]))
        both = normal & (np.minimum(np.abs(y.real), np.abs(y.imag)) > 1e-150)
        assert np.all(np.abs(phase - angle)[both] <= 4 * np.spacing(np.abs(angle[both])))
        on_axis = (y.real == 0) | (y.imag == 0)
        assert np.allclose(phase[on_axis], angle[on_axis], rtol=1e-15, atol=0)
        assert np.array_equal(np.signbit(phase[on_axis]), np.signbit(angle[on_axis]))
    y = np.array([complex(a, b) for a in (inf, -inf, nan, 1.0) for b in (inf, -inf, nan, 2.0)])
    for k in range(len(y)):  # each beside an ordinary value
        amp, phase, top = holo.normalize_polar(np.array([1e-9 + 1e-9j, y[k]]).view(np.float64))
        want = np.hypot(y[k].real, y[k].imag)
        assert top == want or (np.isnan(want) and top < 1e-8)


@pytest.mark.gpu
def test_adjoint_factors_over_all_phases(holo):
    """One target far away: d y / d amp = e^{i phi} e^{i k r} / r, against the same in long double."""
    rng = np.random.default_rng(8)
    n, lam = 4000, 632.8e-9
    phase = rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-60, 12, n)
    phase[:3] = 0.0, -0.0, 1e-300
    amp = rng.uniform(0.5, 1, n)
    u = np.zeros((n, 3))
    u[:, :2] = rng.uniform(-1e-4, 1e-4, (n, 2))
    v = np.array([[0.0, 0.0, 0.4]])
    ga, gp = holo.adjoint(amp, phase, u, v, np.array([0.6, -0.8]), 1, lam, precision="fp64")
    d = v[0] - u
    r = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
    g = complex(0.6, -0.8)
    wave = np.exp(1j * phase) * np.exp(1j * (2 * np.pi / lam) * r) / r
    # k r in FP64: 4e6 rad to 5e-10; the factors themselves are exact to 1e-16
    assert np.max(np.abs(ga - (wave * np.conj(g)).real)) < 4e-9 / 0.4
    assert np.max(np.abs(gp + (amp * wave * np.conj(g)).imag)) < 4e-9 / 0.4

"""The fixed-point FP64 kernel (csrc/fp64_fixed.cuh, variants 6 and 7) against the kernel that runs the
same terms on the FP64 pipe (variant 0), and its host arithmetic against exact values.

Both kernels form bit-equal distances and phases; quotient, sine, cosine and products differ by
less than an ulp of FP64 a term, and variant 0 rounds its running sum once a term: at most
sqrt(N) 2^-53 of the sum for random phases, 1e-14 for the 6000 sources here at the very most."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import LAM, REPO, grid, rel_l2

TOL = 1e-14


def _pair(holo, amp, phase, u, v, sign, kernel=6, lam=LAM):
    return [holo.transform(amp, phase, u, v, sign, lam, precision="fp64", variant=k) for k in (kernel, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [6, 7])
@pytest.mark.parametrize("n,m,layout,sign", [
    (1, 1, "lattice", -1), (63, 513, "lattice", 1), (64, 512, "jitter", -1),
    (65, 2047, "lattice", -1), (1000, 4099, "jitter", 1), (6000, 1500, "lattice", -1),
    (129, 70001, "tilt", 1)])
def test_against_the_fp64_pipe(holo, n, m, layout, sign, kernel):
    rng = np.random.default_rng(n + m)
    u = grid(int(np.ceil(np.sqrt(n))), 10e-6, rng.uniform(0.05, 2.0))[:n]
    v = grid(int(np.ceil(np.sqrt(m))), 7.56e-6, 0.0)[:m]
    if layout != "lattice":  # no coordinate shared between neighbouring targets
        v[:, :2] += rng.uniform(-3e-6, 3e-6, (m, 2))
    if layout == "tilt":
        v[:, 2] = 0.2 * v[:, 0]
    amp, phase = rng.uniform(-1, 1, n), rng.uniform(-10, 10, n)
    a, b = _pair(holo, amp, phase, u, v, sign, kernel)
    assert rel_l2(a, b) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [6, 7])
def test_amplitudes_over_the_whole_range(holo, kernel):
    """Dark, faint and huge sources: each term as exact as the largest of its 64 allows."""
    rng = np.random.default_rng(1)
    u, v = grid(40, 10e-6, 0.35), grid(24, 7.56e-6, 0.0)
    n = len(u)
    phase = rng.uniform(0, 2 * np.pi, n)
    faint = 10.0 ** rng.uniform(-30, 0, n)
    dark = np.where(rng.uniform(size=n) < 0.9, 0.0, 1.0)
    dark[:256] = 0.0
    for amp in (faint, dark, faint * 1e-250, faint * 1e250, np.full(n, 5e-324), np.zeros(n)):
        a, b = _pair(holo, amp, phase, u, v, 1, kernel)
        if not np.any(b):
            assert np.array_equal(a, b)
            continue
        top = np.abs(b).max()  # taken out first: squares of such values leave the FP64 range
        assert rel_l2(a.view(float) / top, b.view(float) / top) < TOL


@pytest.mark.gpu
def test_distances_over_many_scales(holo):
    """Sources from a nanometre to a kilometre from the targets, in one tile and apart."""
    rng = np.random.default_rng(2)
    v = grid(20, 7.56e-6, 0.0)
    z = 10.0 ** rng.uniform(-9, 3, 300)
    u = np.stack([rng.uniform(-1e-3, 1e-3, 300), rng.uniform(-1e-3, 1e-3, 300), z], 1)
    amp, phase = z * rng.uniform(0.5, 1, 300), rng.uniform(0, 2 * np.pi, 300)
    for order in (np.arange(300), np.argsort(z), np.argsort(-z)):
        a, b = _pair(holo, amp[order], phase[order], u[order], v, -1)
        assert rel_l2(a, b) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [6, 7])
def test_coincident_infinite_and_nan_values(holo, kernel):
    """What has no fixed-point form goes through the FP64 operations: the same infinities, NaN
    and finite values as those give."""
    rng = np.random.default_rng(3)
    u, v = grid(10, 10e-6, 0.3), grid(30, 7.56e-6, 0.0)
    amp, phase = rng.uniform(0, 1, 100), rng.uniform(0, 2 * np.pi, 100)
    for edit in ("coincident", "amp_inf", "amp_nan", "phase_nan", "phase_huge", "source_inf",
                 "target_nan"):
        a, p, s, t = amp.copy(), phase.copy(), u.copy(), v.copy()
        if edit == "coincident":
            s[17] = t[100]
        elif edit == "amp_inf":
            a[5] = np.inf
        elif edit == "amp_nan":
            a[70] = np.nan
        elif edit == "phase_nan":
            p[99] = np.nan
        elif edit == "phase_huge":
            p[::7] *= 1e15
        elif edit == "source_inf":
            s[3, 0] = np.inf
        else:
            t[50, 2] = np.nan
        x, y = _pair(holo, a, p, s, t, 1, kernel)
        for f, g in ((x.real, y.real), (x.imag, y.imag)):
            assert np.array_equal(np.isnan(f), np.isnan(g)), edit
            fin = np.isfinite(g)
            assert np.array_equal(f[~fin & ~np.isnan(g)], g[~fin & ~np.isnan(g)]), edit
            assert np.linalg.norm(f[fin] - g[fin]) <= TOL * np.linalg.norm(g[fin]), edit


HOST_CHECK = r"""
#include <cstdio>
#include <cmath>
#include "fp64_tables.h"
using namespace holo;
using namespace holo::fixed;
static uint64_t state = 88172645463325252ull;
static uint64_t next() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static double unit() { return (next() >> 11) * 0x1p-53; }
int main() {
  static TrigEntry trig[kTrigEntries];
  static TurnWords words[kTurnEntries];
  fill_trig(trig);
  fill_turns(words);
  const long double two_pi = 6.283185307179586476925286766559L;
  long bad = 0;
  double trig_err = 0, turn_err = 0, rec_err = 0;
  for (int i = 0; i < 2000000; ++i) {
    double s;  // random, near squares, near powers of two
    if (i % 3 == 0) s = ldexp(1 + unit(), (int)(next() % 60) - 30);
    else if (i % 3 == 1) { const double x = ldexp(floor(ldexp(1 + unit(), 26)), -26); s = x * x * (1 + ((int)(next() % 5) - 2) * 0x1p-52); }
    else s = nextafter(ldexp(1.0, (int)(next() % 20) - 10), (next() & 1) ? 0 : 100);
    const double off = ((int)(next() % 2001) - 1000) * 1e-3 * 0x1p-22;  // the estimate's error
    uint64_t b;
    memcpy(&b, &s, 8);
    const Root r = root((uint32_t)(b >> 32), (uint32_t)b, [&](float x) { return (float)((1.0 / sqrt((double)x)) * (1 + off)); });
    if (ldexp((double)r.d, r.q - 52) != sqrt(s)) ++bad;
    const long double want = 0x1p114L / (long double)r.d;
    rec_err = fmax(rec_err, (double)fabsl((long double)reciprocal(r) - want) * 0x1p-62);
    const double ph = (next() & 1 ? 1 : -1) * ldexp(1 + unit(), (int)(next() % 24));
    memcpy(&b, &ph, 8);
    const uint32_t *k = words[((b >> 52) & 0x7ff) - 1023 - kTurnLow].k;
    const uint64_t t = turns((uint32_t)(b >> 32), (uint32_t)b, k[0], k[1], k[2], k[3]);
    int64_t c, sn;
    const uint32_t index = trig_index(t);
    cos_sin(t, index, trig[index & (kTrigEntries - 1)], &c, &sn);
    const long double a = two_pi * ((long double)(int64_t)t * 0x1p-64L);
    trig_err = fmax(trig_err, fmax((double)fabsl(c * 0x1p-62L - cosl(a)), (double)fabsl(sn * 0x1p-62L - sinl(a))));
    if (fabs(ph) < 4096) {  // beyond, the check's own long double product is no better
      long double d = (long double)ph / two_pi - (long double)(int64_t)t * 0x1p-64L;
      d -= rintl(d);
      turn_err = fmax(turn_err, (double)fabsl(d));
    }
  }
  printf("%ld %.3g %.3g %.3g\n", bad, rec_err, trig_err, turn_err);
  return 0;
}
"""


def test_host_arithmetic(tmp_path):
    """The header's arithmetic on the host: every root correctly rounded whatever the 2^-22
    estimate's error, reciprocals within 2^-60, sines and cosines within 2^-53 (their worst of
    2 million; 1e-17 rms), phases in turns within 2^-50 (2^-61 is what the words hold; the
    check divides in long double, which on x86 has 64 bits)."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    csrc = os.path.join(REPO, "holographic-projector-simulations_gb300", "csrc")
    src = tmp_path / "check.cpp"
    src.write_text(HOST_CHECK)
    exe = tmp_path / "check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", f"-I{csrc}", str(src),
                    os.path.join(csrc, "fp64_tables.cpp"), "-o", str(exe)], check=True)
    bad, rec, trig, turn = subprocess.run([str(exe)], check=True, capture_output=True,
                                          text=True).stdout.split()
    assert int(bad) == 0
    assert float(rec) < 2.0 ** -60 and float(trig) < 2.0 ** -53 and float(turn) < 2.0 ** -50

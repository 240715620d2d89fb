"""A set without points beside one with points: the other set's tile order is still formed, since
chains take it from one plan to the next and batches gather through it."""
import numpy as np
import pytest

from conftest import LAM, grid

pytestmark = pytest.mark.gpu


def _tensor(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64).reshape(-1), device="cuda:0")


@pytest.mark.parametrize("n", [1, 300, 9000])
def test_order_beside_an_empty_set(holo, n):
    pts, none = grid(int(np.ceil(np.sqrt(n))), 10e-6, 0.3)[:n], np.zeros((0, 3))
    want = holo.tile_order(pts)
    with holo.Plan(none, pts) as plan:
        assert np.array_equal(plan.order(1), want) and plan.order(0).size == 0
    with holo.Plan(pts, none) as plan:
        assert np.array_equal(plan.order(0), want) and plan.order(1).size == 0


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("reference_wave", [False, True])
def test_chain_without_sources(holo, on_device, reference_wave):
    """y of no sources is 0, or the reference wave's own modulus and phase; z is the sum over that."""
    none = np.zeros(0)
    v, w = grid(70, 7.56e-6, 0.0), grid(40, 10e-6, 0.35)
    t = _tensor if on_device else (lambda a: np.ascontiguousarray(a).reshape(-1))
    back = (lambda a: a.cpu().numpy()) if on_device else np.asarray
    ya, yp, za, zp = (back(a) for a in holo.project(t(none), t(none), t(none), t(v), t(w), LAM,
                                                    reference_wave=reference_wave))
    if not reference_wave:
        assert not ya.any() and not yp.any() and not za.any()
        return
    z = np.asarray(holo.transform(ya, yp, v, w, 1, LAM, precision="fp64"))
    z = z / np.abs(z).max() if np.abs(z).max() >= 1e-6 else z
    got = za * np.exp(1j * zp)
    assert np.linalg.norm(got - z) <= 1e-5 * max(np.linalg.norm(z), 1e-30)


def test_batch_with_empty_problems(holo):
    import torch
    rng = np.random.default_rng(0)
    u, v, none = grid(40, 10e-6, 0.3), grid(50, 7.56e-6, 0.0), np.zeros((0, 3))
    amp, phase = rng.uniform(0, 1, len(u)), rng.uniform(0, 2 * np.pi, len(u))
    y = [torch.full((2 * k,), 7.0, dtype=torch.float64, device="cuda:0") for k in (0, len(v), len(v))]
    # the sources of a problem without targets are still gathered
    problems = [holo.Problem(_tensor(amp), _tensor(phase), _tensor(u), _tensor(none), 1, LAM, y[0]),
                holo.Problem(_tensor(none), _tensor(none), _tensor(none), _tensor(v), 1, LAM, y[1]),
                holo.Problem(_tensor(amp), _tensor(phase), _tensor(u), _tensor(v), 1, LAM, y[2])]
    with holo.Batch(problems) as batch:
        batch.execute()
    torch.cuda.synchronize()
    want = np.asarray(holo.transform(amp, phase, u, v, 1, LAM, precision="fp64"))
    got = y[2].cpu().numpy().view(complex)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)

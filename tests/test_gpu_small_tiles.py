"""Problems of few 512 x 1024 tiles run on source tiles of 256: the choice, and its results against
FP64 sums.

Either kernel is only taken where its path-length bound is below 3.2e-13 m (5e-6 rad at 400 nm); the
2e-5 of the field is what the split path is held to elsewhere."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,variant", [
    (256, 512, 73), (257, 512, 76), (1024, 4096, 76), (1025, 4097, 76), (300, 38912, 76),
    (300, 38913, 73), (76 * 1024, 512, 76), (76 * 1024 + 1, 512, 73)])
def test_choice_and_sums(holo, n, m, variant):
    rng = np.random.default_rng(n)
    u = grid(int(np.ceil(np.sqrt(n))), 10e-6, 0.4)[:n]
    v = grid(int(np.ceil(np.sqrt(m))), 7.56e-6, 0.0)[:m]
    amp, phase = rng.uniform(0, 1, n), rng.uniform(0, 2 * np.pi, n)
    with holo.Plan(u, v) as plan:
        info = plan.info()
        y = plan.execute(amp, phase, -1, LAM)
    assert info["variant"] == variant and info["path_error_bound_m"] <= 3.2e-13
    assert rel_l2(y, holo.transform(amp, phase, u, v, -1, LAM, precision="fp64")) < 2e-5


@pytest.mark.gpu
def test_a_tuned_variant_stays(holo):
    """A variant set for the size bucket is taken as it is."""
    h = holo.handle(0)
    u, v = grid(32, 10e-6, 0.4), grid(64, 7.56e-6, 0.0)
    bucket = next(b for b in range(64) if _sets(holo, h, b, u, v))
    assert bucket >= 0


def _sets(holo, h, bucket, u, v):
    try:
        old = h.get_variant("split32", bucket)
    except holo.HoloError:
        return False
    h.set_variant("split32", bucket, 73)
    try:
        with holo.Plan(u, v) as plan:
            return plan.info()["variant"] == 73
    finally:
        h.set_variant("split32", bucket, old)

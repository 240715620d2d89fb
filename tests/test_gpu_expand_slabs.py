"""A sum by cluster expansions whose coefficients take more scratch than one launch gets: its target
clusters in slabs, on its own and in a batch, against the FP64 kernel on a sample of the targets."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2

pytestmark = pytest.mark.gpu

TOL = 2.5e-6  # as for sums in one slab


def test_more_than_one_slab(holo):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")
    rng = np.random.default_rng(11)
    u, v = grid(2048, 10e-6, 0.5), grid(2050, 7.56e-6, 0.0)
    n, m = len(u), len(v)
    amp, phase = rng.uniform(0, 1, n), rng.uniform(0, 2 * np.pi, n)
    a, p, tu, tv = t(amp), t(phase), t(u), t(v)
    with holo.Plan(tu, tv, "split32") as plan:
        n0 = holo.api.kernel_launches()
        y = plan.execute(a, p, -1, LAM)
        launches = holo.api.kernel_launches() - n0
    assert launches >= 9, launches  # gather, then four launches a slab
    idx = np.unique(np.concatenate([np.arange(200), np.arange(m - 200, m),
                                    rng.choice(m, 1500, replace=False)]))
    want = holo.transform(a, p, tu, t(v[idx]), -1, LAM, precision="fp64").cpu().numpy()
    assert rel_l2(y.cpu().numpy()[idx], want) < TOL
    out = [torch.zeros(2 * m, dtype=torch.float64, device="cuda:0") for _ in range(2)]
    with holo.Batch([holo.Problem(a, p, tu, tv, -1, LAM, o) for o in out]) as batch:
        batch.execute()
        batch.execute()
    torch.cuda.synchronize()
    for o in out:
        got = torch.view_as_complex(o.view(-1, 2)).cpu().numpy()[idx]
        assert rel_l2(got, want) < TOL

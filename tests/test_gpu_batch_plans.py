"""A batch is replayed: the problems that it runs pair by pair are tiled as a plan to keep is."""
import numpy as np
import pytest

from conftest import LAM, grid

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")


@pytest.mark.parametrize("n,m,tilt", [(20000, 150000, 0.1), (40000, 40000, 0.3), (30000, 3000, 0.1)])
def test_packed_tiles_where_a_plan_packs(holo, n, m, tilt):
    import torch
    rng = np.random.default_rng(n)
    u = grid(int(np.ceil(np.sqrt(n))), 10e-6, 0.35)[:n]
    v = grid(int(np.ceil(np.sqrt(m))), 7.56e-6, 0.0)[:m]
    u[:, 2] += tilt * u[:, 0]  # no cluster expansions
    a, p, tu, tv = _t(rng.uniform(0, 1, n)), _t(rng.uniform(0, 2 * np.pi, n)), _t(u), _t(v)
    n0 = holo.api.kernel_launches()
    with holo.Plan(tu, tv) as plan:
        planning = holo.api.kernel_launches() - n0
        assert plan.tiling()["sources"] == "packed", plan.info()
        y = plan.execute(a, p, 1, LAM)
    out = torch.zeros(2 * m, dtype=torch.float64, device="cuda:0")
    n0 = holo.api.kernel_launches()
    with holo.Batch([holo.Problem(a, p, tu, tv, 1, LAM, out)]) as batch:
        assert holo.api.kernel_launches() - n0 >= planning  # the same sorts, then the captured ones
        batch.execute()
    torch.cuda.synchronize()
    assert torch.linalg.norm(torch.view_as_complex(out.view(-1, 2)) - y) < 1e-5 * torch.linalg.norm(y)

"""A tuned kernel variant of any source tile leaves a sum its cluster expansions."""
import numpy as np
import pytest

from conftest import LAM, grid, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [256, 512, 768, 1024])
@pytest.mark.parametrize("n,m", [(16384, 262144), (65536, 65536), (16385, 131073)])
def test_expansions_on_tuned_tiles(holo, tile, n, m):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")
    variant = next(v["variant"] for v in holo.variants("split32")
                   if v["source_tile"] == tile and v["pair_loop"] == 3)
    rng = np.random.default_rng(n)
    u = grid(int(np.ceil(np.sqrt(n))), 10e-6, 0.35)[:n]
    v = grid(int(np.ceil(np.sqrt(m))), 7.56e-6, 0.0)[:m]
    amp, phase = rng.uniform(0, 1, n), rng.uniform(0, 2 * np.pi, n)
    h, bucket = holo.handle(0), holo.size_bucket(n, m)
    old = h.get_variant("split32", bucket)
    h.set_variant("split32", bucket, variant)
    try:
        with holo.Plan(t(u), t(v)) as plan:
            if plan.info()["source_tile"] != tile:
                pytest.skip("the error bound rules these tiles out")
            n0 = holo.api.kernel_launches()
            y = plan.execute(t(amp), t(phase), 1, LAM).cpu().numpy()
            assert holo.api.kernel_launches() - n0 in (5, 6)
    finally:
        h.set_variant("split32", bucket, old)
    idx = np.unique(np.concatenate([np.arange(min(m, 300)), np.arange(0, m, 211)]))
    want = holo.transform(amp, phase, u, v[idx], 1, LAM, precision="fp64")
    assert rel_l2(y[idx], want) < 2.5e-6

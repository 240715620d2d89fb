"""Device memory that a batch holds: sums by cluster expansions that need slabs of scratch run one
after another and share it, and the rest share a bounded one."""
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
import numpy as np
import torch
sys.path.insert(0, ".")
import __graft_entry__
from tests.conftest import LAM, grid
holo = __graft_entry__.load_package()
n_side, m_side, count = (int(a) for a in sys.argv[1:4])
t = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda:0")
rng = np.random.default_rng(0)
u, v = grid(n_side, 10e-6, 0.5), grid(m_side, 7.56e-6, 0.0)
a, p, tu, tv = t(rng.uniform(0, 1, len(u))), t(rng.uniform(0, 6, len(u))), t(u), t(v)
y = [torch.zeros(2 * len(v), dtype=torch.float64, device="cuda:0") for _ in range(count)]
problem = lambda i: holo.Problem(a, p, tu, tv, -1, LAM, y[i])
free = lambda: torch.cuda.mem_get_info(0)[0]
with holo.Batch([problem(0)]) as batch:  # loads the kernels
    batch.execute()
torch.cuda.synchronize()
one = holo.Batch([problem(0)])
before = free()
many = holo.Batch([problem(i) for i in range(count)])
many.execute()
torch.cuda.synchronize()
held = before - free()
assert all(torch.equal(z, y[0]) for z in y) and y[0].any()
print("HELD", held / 2**20)
"""


# (sides of the source and target planes, problems, most MiB that one batch of them may hold: the
# plans' part is 0.5, 0.1 and 0.2 GiB a problem, the shared scratch up to 4 GiB)
@pytest.mark.parametrize("n_side,m_side,count,most", [
    (2048, 2050, 6, 4096),     # slabs, 5.0 GiB when each held its own scratch
    (700, 1400, 40, 8192),     # slabs of a part of the GPU, 23.0 GiB
    (300, 2048, 40, 14336)])   # one slab each, two rounds, 15.3 GiB
def test_memory_held(built, n_side, m_side, count, most):
    out = subprocess.run([sys.executable, "-c", SCRIPT, str(n_side), str(m_side), str(count)], cwd=REPO,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    held = float(out.stdout.split("HELD")[1])
    assert held < most

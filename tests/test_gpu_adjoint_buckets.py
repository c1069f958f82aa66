"""Which buckets have the reverse mode, at the ends of its range: its staging against the space of the phases.

Stokes quads of k = 1 with 20 test dofs (the staging is larger than the phases' own tables), with 80, and of
k = 3 with 155 (one CTA's shared memory nearly full), each on 16 warps and, where it is small, on 8.  The
gradient is compared with the extended-precision hand gradient at 1e-8, the bound of the other
reverse-mode tests: the coefficients are loads, so it is linear in X = G^-1 B, whose error at
cells of h = 1/2 is the forward's (below 1e-10)."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402
from tests.helpers import coeffs_for, stokes2d  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,dk", [(1, 0), (1, 1), (3, 1)])
def test_reverse_mode_of_small_and_full_buckets(k, dk, oracle_mod):
    _, bucket, nodes, par = stokes2d(k, dk)
    X = oracle_mod.OraclePlan(bucket, xp=True)
    plan = dlib.Plan(bucket)
    n, M = nodes.shape[0], plan.info["M"]
    co = coeffs_for(bucket, plan.info, n)
    rng = np.random.default_rng(4)
    r, lb = rng.normal(size=(n, M)), rng.normal(size=(n, M))
    Kb = r[:, :, None] * r[:, None, :]
    ref = X.adjoint(nodes, par, co, Kb, lb, nthreads=os.cpu_count() or 1)
    for C in (n, torch.cuda.get_device_properties(0).multi_processor_count + 1):
        i = np.arange(C) % n
        got, info = plan.adjoint(*(torch.as_tensor(np.ascontiguousarray(a[i])).cuda() for a in (nodes, par, co, Kb, lb)))
        torch.cuda.synchronize()
        assert int(info.abs().max()) == 0
        got = got.cpu().numpy()
        for c in range(n):
            assert np.linalg.norm(got[c] - ref[c]) <= 1e-8 * np.linalg.norm(ref[c])
        assert np.array_equal(got, got[i])

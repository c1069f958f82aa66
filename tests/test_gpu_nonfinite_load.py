"""A load that is not finite in one cell (an infinity at every point, one NaN) reaches that cell's F, l and s and
nothing else: G, B, K, S, W and info are those of the same call with a finite load, bit for bit.  K = B^T G^-1 B does not
hold the load; the buckets place the load's column differently among the trial columns (alone in its tile,
last in the traces' tile), and large buckets run a cluster or a CTA per cell."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402
from tests.helpers import coeffs_for, poisson2d, poisson3d, stokes2d, stokes_tri  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(x):
    return torch.as_tensor(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("make", [lambda: poisson2d(2, 2), lambda: poisson2d(4, 2), lambda: poisson3d(2, 1),
                                  lambda: stokes2d(2, 2), lambda: poisson2d(5, 2), lambda: stokes_tri(4, 2),
                                  lambda: stokes2d(3, 2), lambda: stokes2d(6, 2), lambda: stokes_tri(6, 2)])
@pytest.mark.parametrize("C", [4, 80, 160])
def test_load_that_is_not_finite(make, C):
    _, bucket, nodes, par = make()
    plan = dlib.Plan(bucket)
    i = np.arange(C) % nodes.shape[0]
    nodes, par, co = nodes[i], par[i], coeffs_for(bucket, plan.info, C)
    bad = co.copy()
    bad[1] = np.inf
    bad[2, 0, plan.info["Q_G"] + 1] = np.nan  # a volume point of B and F
    hit = np.isin(np.arange(C), (1, 2))

    def calls(c):
        cells = (_dev(nodes), _dev(par), _dev(c))
        out, (G, B, F), (W, y, info) = plan.assemble(*cells), plan.parts(*cells), plan.dls(*cells)
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (out["K"], out["S"], out["info"], G, B, W, info)], \
               [t.cpu().numpy() for t in (out["l"], out["s"], F, y)]

    (same, load), (ref_same, ref_load) = calls(bad), calls(co)
    assert (ref_same[2] == 0).all()
    for a, b in zip(same, ref_same):
        assert np.array_equal(a, b)
    for a, b in zip(load, ref_load):
        assert np.array_equal(a[~hit], b[~hit])
        assert not np.isfinite(a[hit]).all(axis=1).any()

"""The scatter plan's apply stages a cell's S where its map names enough of the rows, and gathers the entries
otherwise.  Both sides of each line against a dense accumulation (sums of a few O(1) products in another order:
1e-13), maps with empty rows, with several entries per row and with weights.  A map of a few of very many rows must be
gathered: S does not fit, whatever the product of its sizes is modulo 2^32."""
import ctypes as ct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(x):
    return None if x is None else torch.as_tensor(np.ascontiguousarray(x)).cuda()


def _staged(plan):
    return dlib.load().dpg_debug_scatter_staged(plan.h)


# (t, rows with entries, entries per row): S of 5, 20, 49, 49, 65 and 71 KB
@pytest.mark.parametrize("t,rows,fan,staged", [
    (26, 26, 1, 1), (26, 8, 1, 1), (26, 7, 1, 0), (26, 3, 3, 1), (50, 15, 1, 1), (50, 14, 1, 0), (78, 35, 1, 1),
    (78, 34, 1, 0), (78, 18, 2, 1), (78, 1, 1, 0), (91, 70, 1, 1), (91, 60, 1, 0), (95, 72, 1, 1), (95, 20, 3, 0)])
@pytest.mark.parametrize("weights", [False, True])
def test_both_sides_of_the_lines(t, rows, fan, staged, weights):
    C = 7
    rng = np.random.default_rng(t + rows)
    named = np.zeros((C, t), bool)
    for c in range(C):
        named[c, rng.choice(t, rows, replace=False)] = True
    ptr = np.concatenate([[0], np.cumsum(named.reshape(-1) * fan)]).astype(np.int64)
    n = C * rows + 5
    gid = np.concatenate([rng.choice(n, rows * fan, replace=False) if rows * fan <= n else rng.integers(0, n, rows * fan)
                          for _ in range(C)]).astype(np.int64)
    w = rng.normal(size=len(gid)) if weights else None
    S, s = rng.normal(size=(C, t, t)), rng.normal(size=(C, t))
    A, b = np.zeros((n, n)), np.zeros(n)
    for c in range(C):
        P = np.zeros((t, n))
        for a in range(t):
            for k in range(ptr[c * t + a], ptr[c * t + a + 1]):
                P[a, gid[k]] += 1.0 if w is None else w[k]
        A += P.T @ S[c] @ P
        b += P.T @ s[c]
    row_ptr = np.arange(0, n * n + 1, n, dtype=np.int64)  # a full graph
    col = np.tile(np.arange(n), n).astype(np.int64)
    plan = dlib.ScatterPlan(C, t, _dev(ptr), _dev(gid), _dev(w), n, _dev(row_ptr), _dev(col))
    assert _staged(plan) == staged
    values = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    rhs = torch.zeros(n, dtype=torch.float64, device="cuda")
    plan.apply(_dev(S), _dev(s), values, rhs)
    torch.cuda.synchronize()
    assert int(plan.missing) == 0
    assert np.abs(values.cpu().numpy().reshape(n, n) - A).max() <= 1e-13 * max(1.0, np.abs(A).max())
    assert np.abs(rhs.cpu().numpy() - b).max() <= 1e-13 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("t", [46341, 65536])
def test_few_rows_of_very_many_are_gathered(t):
    ptr = np.zeros(t + 1, np.int64)
    ptr[1:] = 1
    ptr[-1] = 2  # entries in the first and the last row
    plan = dlib.ScatterPlan(1, t, _dev(ptr), _dev(np.array([0, 1])), None, 2, _dev(np.array([0, 2, 4])),
                            _dev(np.array([0, 1, 0, 1])))
    assert int(plan.missing) == 0
    assert _staged(plan) == 0

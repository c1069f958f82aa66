"""Kernel variants and launch shapes at the sizes where they can go wrong.

  * Small buckets (two 8-warp CTAs per SM) against the work queue's 16-warp CTAs, bit for bit: the phases
    and their sums do not depend on the warps; one cell, fewer and more cells than CTAs.
  * Test vars with an odd number of 8-row tiles, F inside or behind the traces' last tile: the oracle.
  * Large buckets with a cluster of CTAs per cell (few cells) against one CTA per cell, bit for bit.
  * The host pipeline across a chunk's end, bit for bit against one device call.
  * Recovery with 3 to 32 and more field dofs against dense solves of well conditioned matrices
    (condition below 100, so 1e-12 is a hundred times the rounding of either solve).
  * The scatter plan's staged apply: one dof, an odd S (unaligned cells), dofs shared within a cell, and
    a cell too large to stage, against a dense accumulation (sums of at most a few dozen O(1)
    products in another order: 1e-13).
  * K = B G^-1 B^T for every number of trial tiles (how its blocks are dealt out depends on it) against
    dense solves: condition below 10, 125 test rows, so 1e-12 is ten times 125 roundings at that
    condition."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402
from tests.helpers import (cdr2d, check_against_truth, coeffs_for, poisson2d, poisson3d, poisson_tri,  # noqa: E402
                           stokes2d, stokes_tri)

pytestmark = pytest.mark.gpu

KEYS = ("K", "l", "S", "s", "info")


def _dev(x):
    return None if x is None else torch.as_tensor(np.ascontiguousarray(x)).cuda()


def _cells(make, C, seed=3):
    """C cells: the mesh's cells again and again, every cell with its own coefficients."""
    form, bucket, nodes, par = make()
    plan = dlib.Plan(bucket)
    idx = np.arange(C) % nodes.shape[0]
    return bucket, plan, nodes[idx], par[idx], coeffs_for(bucket, plan.info, C, seed=seed)


SMALL = [lambda: poisson2d(1, 1), lambda: poisson2d(2, 2), lambda: poisson2d(3, 2), lambda: cdr2d(3, 2),
         lambda: poisson_tri(1, 2), lambda: poisson_tri(4, 2), lambda: stokes2d(1, 2), lambda: stokes_tri(2, 2),
         lambda: poisson3d(1, 1)]


@pytest.mark.parametrize("make", SMALL)
@pytest.mark.parametrize("C", [1, 299])
def test_small_buckets_equal_the_queue(make, C):
    _, plan, nodes, par, co = _cells(make, C)
    nodes, par, co = _dev(nodes), _dev(par), _dev(co)
    ref = plan.assemble(nodes, par, co)
    out = {k: v.fill_(7) for k, v in plan.alloc_outputs(C).items()}
    dlib.assemble_multi([(plan, nodes, par, co, out)])
    torch.cuda.synchronize()
    for k in KEYS:
        assert torch.equal(out[k], ref[k]), k


@pytest.mark.parametrize("make", [lambda: poisson2d(2, 1), lambda: poisson2d(2, 2), lambda: poisson2d(4, 2, 2, 2),
                                  lambda: poisson_tri(3, 2), lambda: cdr2d(2, 1), lambda: stokes2d(2, 2, 2, 1),
                                  lambda: poisson3d(1, 1)])
def test_odd_tiles_match_the_oracle(make):
    from oracle import oracle
    bucket, plan, nodes, par, co = _cells(make, make()[2].shape[0])
    out = plan.assemble(_dev(nodes), _dev(par), _dev(co))
    torch.cuda.synchronize()
    ref = oracle.OraclePlan(bucket).assemble(nodes, par, co)
    got = {k: out[k].cpu().numpy() for k in KEYS}
    assert (got["info"] == 0).all()
    check_against_truth(oracle, bucket, nodes, par, co, got, ref)


@pytest.mark.parametrize("make", [lambda: stokes2d(3, 2, 2, 2, 0.1), lambda: stokes2d(6, 2, 2, 1, 0.1),
                                  lambda: stokes_tri(4, 2)])
@pytest.mark.parametrize("C", [1, 3, 41])
def test_cluster_per_cell_equals_one_cta(make, C):
    _, plan, nodes, par, co = _cells(make, 80)  # 80 cells: a CTA per cell
    nodes, par, co = _dev(nodes), _dev(par), _dev(co)
    x = torch.linspace(-1, 1, 80 * plan.info["M"], dtype=torch.float64, device="cuda").reshape(80, -1)
    few = (nodes[:C].contiguous(), par[:C].contiguous(), co[:C].contiguous())
    ref, out = plan.assemble(nodes, par, co), plan.assemble(*few)
    e_ref, e = plan.energy_error(nodes, par, co, x)[0], plan.energy_error(*few, x[:C])[0]
    w_ref, w = plan.dls(nodes, par, co)[0], plan.dls(*few)[0]
    torch.cuda.synchronize()
    for k in KEYS:
        assert torch.equal(out[k], ref[k][:C]), k
    assert torch.equal(w, w_ref[:C])
    assert torch.allclose(e, e_ref[:C], rtol=1e-12, atol=0.0)  # its sum's order follows the threads


@pytest.mark.parametrize("C", [591, 593])
def test_host_pipeline_across_chunks(C):
    _, plan, nodes, par, co = _cells(lambda: poisson3d(2, 1, 2, 0.1), C)
    ref = plan.assemble(_dev(nodes), _dev(par), _dev(co))
    torch.cuda.synchronize()
    out = plan.assemble_host(nodes, par, co)
    for k in KEYS:
        assert np.array_equal(out[k], ref[k].cpu().numpy()), k


# 3, 7, 9, 12, 27, 28, 32 fields: one to four tiles, whole and ragged; 42: the block kernel
@pytest.mark.parametrize("make", [lambda: poisson2d(1, 1), lambda: stokes2d(1, 2), lambda: poisson_tri(2, 2),
                                  lambda: poisson2d(2, 2), lambda: poisson2d(3, 2), lambda: stokes2d(2, 2),
                                  lambda: poisson3d(2, 1), lambda: stokes_tri(3, 2)])
def test_recovery_sizes(make):
    plan = dlib.Plan(make()[1])
    nf, M, C = plan.info["n_field"], plan.info["M"], 37
    rng = np.random.default_rng(nf)
    X = rng.normal(size=(C, M, 4 * M))
    K = X @ X.transpose(0, 2, 1) / (4 * M)
    l, t = rng.normal(size=(C, M)), rng.normal(size=(C, M - nf))
    u, info = plan.recover_fields(_dev(K), _dev(l), _dev(t))
    torch.cuda.synchronize()
    assert int(info.abs().max()) == 0
    ref = np.linalg.solve(K[:, :nf, :nf], (l[:, :nf] - np.einsum("cij,cj->ci", K[:, :nf, nf:], t))[:, :, None])[:, :, 0]
    u = u.cpu().numpy()
    assert np.array_equal(u[:, nf:], t)
    assert np.linalg.norm(u[:, :nf] - ref) <= 1e-12 * np.linalg.norm(ref)


def _ring_map(C, t, share):
    """Local dof a of cell c -> global dof c (t - share) + a: neighbours share `share` dofs, and the last
    dof of a cell repeats its first one (two local dofs on one global dof)."""
    gid = (np.arange(C)[:, None] * max(1, t - share) + np.arange(t)[None, :]).astype(np.int64)
    if t > 2:
        gid[:, -1] = gid[:, 0]
    return gid, int(gid.max()) + 1


@pytest.mark.parametrize("C,t,share", [(3, 1, 0), (5, 5, 2), (40, 13, 3), (7, 78, 9), (3, 130, 4)])
def test_scatter_plan_sizes(C, t, share):
    gid, n = _ring_map(C, t, share)
    rng = np.random.default_rng(t)
    S, s = rng.normal(size=(C, t, t)), rng.normal(size=(C, t))
    A, b = np.zeros((n, n)), np.zeros(n)
    for c in range(C):
        np.add.at(A, (gid[c][:, None], gid[c][None, :]), S[c])
        np.add.at(b, gid[c], s[c])
    touched = np.zeros((n, n), bool)
    for c in range(C):
        touched[np.ix_(gid[c], gid[c])] = True
    rows, cols = np.nonzero(touched)
    row_ptr = np.zeros(n + 1, np.int64)
    np.add.at(row_ptr, rows + 1, 1)
    row_ptr = np.cumsum(row_ptr)
    plan = dlib.ScatterPlan(C, t, _dev(np.arange(C * t + 1, dtype=np.int64)), _dev(gid.reshape(-1)), None, n,
                            _dev(row_ptr), _dev(cols.astype(np.int64)))
    values = torch.zeros(len(cols), dtype=torch.float64, device="cuda")
    rhs = torch.zeros(n, dtype=torch.float64, device="cuda")
    plan.apply(_dev(S), _dev(s), values, rhs)
    torch.cuda.synchronize()
    assert int(plan.missing) == 0
    assert np.abs(values.cpu().numpy() - A[rows, cols]).max() <= 1e-13 * max(1.0, np.abs(A).max())
    assert np.abs(rhs.cpu().numpy() - b).max() <= 1e-13 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("M", [1, 9, 17, 25, 33, 41, 49, 57, 65, 73, 81, 89, 97, 105, 112])
def test_gram_of_the_solution_for_every_number_of_trial_tiles(M):
    rng = np.random.default_rng(M)
    C, N = 5, 125
    A = rng.standard_normal((C, N, N))
    G = A @ A.transpose(0, 2, 1) / N + np.eye(N)
    B, F = rng.standard_normal((C, M, N)), rng.standard_normal((C, N))
    K, l, info = dlib.factoredCholeskySolve(_dev(G), _dev(B), _dev(F))
    X = np.linalg.solve(G, np.concatenate([B, F[:, None]], 1).transpose(0, 2, 1))
    Kx, lx = B @ X[:, :, :M], (B @ X[:, :, M:])[:, :, 0]
    assert (info.cpu().numpy() == 0).all()
    assert np.abs(K.cpu().numpy() - Kx).max() <= 1e-12 * np.abs(Kx).max()
    assert np.abs(l.cpu().numpy() - lx).max() <= 1e-12 * np.abs(Kx).max()

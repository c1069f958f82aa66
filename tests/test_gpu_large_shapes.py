"""Launch shapes of the large buckets and of the calls around them.

  * G, B, F and a failed factorisation with a CTA per cell (more cells than half the SMs) and with a cluster per
    cell (fewer): the same bits, and the oracle's info.
  * A graph whose large buckets share one workspace and run one after another: the bits of their own calls, at
    every replay.
  * A call captured by the caller, with clusters and with single CTAs.
  * The host pipeline over three and more chunks, so that a buffer is used again while its copies out may still run,
    bit for bit against one device call."""
import ctypes as ct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402
from tests.helpers import coeffs_for, poisson2d, poisson3d, stokes2d, stokes_tri  # noqa: E402

pytestmark = pytest.mark.gpu

KEYS = ("K", "l", "S", "s", "info")


def _dev(x):
    return None if x is None else torch.as_tensor(np.ascontiguousarray(x)).cuda()


def _team(plan, C):
    """CTAs per cell"""
    out = (ct.c_int * 5)()
    assert dlib.load().dpg_debug_launch_shape(plan.h, 0, C, out) == 0
    return out[2]


def _cells(make, C, seed=3):
    """C cells: the mesh's cells again and again, every cell with its own coefficients."""
    _, bucket, nodes, par = make()
    plan = dlib.Plan(bucket)
    i = np.arange(C) % nodes.shape[0]
    return bucket, plan, nodes[i], par[i], coeffs_for(bucket, plan.info, C, seed=seed)


LARGE = [lambda: stokes2d(3, 2, 2, 2, 0.1), lambda: stokes2d(6, 2, 2, 1, 0.1), lambda: stokes_tri(4, 2)]


@pytest.mark.parametrize("make", LARGE)
def test_cta_per_cell_equals_a_cluster_per_cell(make, oracle_mod):
    C, few, bad = 80, 7, 5
    bucket, plan, nodes, par, co = _cells(make, C)
    assert _team(plan, C) == 1 and _team(plan, few) > 1 and _team(plan, 41) > 1
    nodes[bad, :, 0] = -nodes[bad, :, 0]  # det J < 0
    cells = (_dev(nodes), _dev(par), _dev(co))
    some = tuple(t[:few].contiguous() for t in cells)
    parts, out = plan.parts(*cells), plan.assemble(*cells)
    p_few, o_few = plan.parts(*some), plan.assemble(*some)
    torch.cuda.synchronize()
    for a, b in zip(parts, p_few):
        assert torch.equal(a[:few], b)
    info = oracle_mod.OraclePlan(bucket).assemble(nodes[:few], par[:few], co[:few])["info"]
    assert info[bad] != 0 and np.array_equal(o_few["info"].cpu().numpy(), info)
    assert np.array_equal(out["info"].cpu().numpy(), np.where(np.arange(C) == bad, info[bad], 0))
    keep = [c for c in range(few) if c != bad]
    for k in KEYS:
        assert torch.equal(out[k][keep], o_few[k][keep]), k


def test_graph_with_one_shared_workspace():
    items = []
    for make, C in ((LARGE[0], 90), (LARGE[1], 9), (LARGE[2], 40), (lambda: poisson2d(2, 2), 200),
                    (lambda: poisson3d(2, 1), 30)):
        _, plan, nodes, par, co = _cells(make, C)
        items.append((plan, _dev(nodes), _dev(par), _dev(co), plan.alloc_outputs(C)))
    arr, L = dlib._batches(items), dlib.load()
    L.dpg_debug_graph_capture_shared.argtypes = L.dpg_graph_capture.argtypes
    h = ct.c_void_p()
    assert L.dpg_debug_graph_capture_shared(len(items), ct.cast(arr, ct.c_void_p), 0, ct.byref(h)) == 0
    for _ in range(3):
        for _, _, _, co, out in items:
            co.mul_(1.25)
            for k in KEYS:
                out[k].fill_(7)
        L.dpg_graph_launch(h, dlib._stream_ptr(None))
        torch.cuda.synchronize()
        for plan, n, q, c, out in items:
            ref = plan.assemble(n, q, c)
            for k in KEYS:
                assert torch.equal(out[k], ref[k]), k
    L.dpg_graph_destroy(h)


@pytest.mark.parametrize("make,C", [(LARGE[0], 5), (LARGE[0], 80), (lambda: poisson2d(2, 2), 5),
                                    (lambda: poisson2d(2, 2), 200)])
def test_captured_by_the_caller(make, C):
    _, plan, nodes, par, co = _cells(make, C)
    nodes, par, co = _dev(nodes), _dev(par), _dev(co)
    out = plan.alloc_outputs(C)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.assemble(nodes, par, co, out)
    co.mul_(1.5)
    for _ in range(2):
        for k in KEYS:
            out[k].fill_(7)
        g.replay()
        torch.cuda.synchronize()
        ref = plan.assemble(nodes, par, co)
        for k in KEYS:
            assert torch.equal(out[k], ref[k]), k


# chunks of whole waves, about 64 MB of outputs: with all outputs five of 592 hexes and a rest, three of 296 quads and a rest
@pytest.mark.parametrize("make,C", [(lambda: poisson3d(2, 1, 2, 0.1), 5 * 592 + 5), (lambda: stokes2d(4, 2, 2, 2, 0.1), 900)])
@pytest.mark.parametrize("flags", [0, 1, 2])
def test_host_pipeline_over_many_chunks(make, C, flags):
    _, plan, nodes, par, co = _cells(make, C)
    ref = plan.assemble(_dev(nodes), _dev(par), _dev(co))
    torch.cuda.synchronize()
    M, t = plan.info["M"], plan.info["n_trace"]
    out = dict(K=np.full((C, M, M), 7.0), l=np.full((C, M), 7.0), S=np.full((C, t, t), 7.0), s=np.full((C, t), 7.0),
               info=np.full(C, 7, np.int32))
    plan.assemble_host(nodes, par, co, out, flags=flags)
    for k in KEYS:
        if k in ("Kl", "Ss")[flags - 1] and flags:
            assert (out[k] == 7.0).all(), k
        else:
            assert np.array_equal(out[k], ref[k].cpu().numpy()), k

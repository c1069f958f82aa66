"""The Gram phase's ring of staged chunks: one to four stages of 4, 8 or 16 points.

The points are summed in the same order and joined every 32 whatever the chunk, so a plan on the ring of 4-point
chunks gives the bits of the ring that its plan was made with.  Rings by kernel: one, two and four stages in 2D and
3D, on 8 warps and on 16.  Buckets whose shared memory holds the 4-point ring only, against the oracle."""
import ctypes as ct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402
from tests.helpers import cdr2d, check_against_truth, coeffs_for, poisson2d, poisson3d, stokes2d, stokes_tri  # noqa: E402

pytestmark = pytest.mark.gpu


def _dev(x):
    return None if x is None else torch.as_tensor(np.ascontiguousarray(x)).cuda()


def ring(plan):
    """(points per chunk, stages)"""
    out = (ct.c_int * 5)()
    assert dlib.load().dpg_debug_launch_shape(plan.h, 0, 1, out) == 0
    return tuple(out[3:])


@pytest.mark.parametrize("make,first,second", [
    (lambda: poisson2d(1, 1), (16, 1), (4, 2)), (lambda: poisson2d(2, 2), (16, 2), (4, 4)),
    (lambda: cdr2d(3, 2), (8, 2), (4, 4)), (lambda: poisson2d(4, 2), (16, 2), (4, 4)),
    (lambda: poisson3d(1, 1), (16, 2), (4, 4)), (lambda: poisson3d(2, 1), (8, 2), (4, 4)),
    (lambda: stokes2d(2, 2), (8, 2), (4, 4)), (lambda: stokes2d(1, 0), (16, 1), (4, 1))])
def test_ring_of_4_point_chunks_gives_the_same_bits(make, first, second):
    _, bucket, nodes, par = make()
    plan = dlib.Plan(bucket)
    C, M = 160, plan.info["M"]  # two waves of 16-warp CTAs, one of 8-warp ones
    i = np.arange(C) % nodes.shape[0]
    cells = (_dev(nodes[i]), _dev(par[i]), _dev(coeffs_for(bucket, plan.info, C)))
    Kb = torch.randn((C, M, M), dtype=torch.float64, device="cuda")

    def calls():
        out = []
        for n in (37, C):
            few = tuple(None if t is None else t[:n] for t in cells)
            out += list(plan.assemble(*few).values()) + list(plan.parts(*few)) + list(plan.dls(*few))
            out += list(plan.adjoint(*few, Kb[:n])) if few[2] is not None else []
        torch.cuda.synchronize()
        return out

    assert ring(plan) == first
    ref = calls()
    assert dlib.load().dpg_debug_set_gram_chunk(plan.h, 4) == 0
    assert ring(plan) == second
    for a, b in zip(calls(), ref):
        assert torch.equal(a, b)


@pytest.mark.parametrize("make", [lambda: stokes_tri(2, 4), lambda: stokes_tri(3, 3)])
def test_buckets_of_the_4_point_ring_match_the_oracle(make, oracle_mod):
    _, bucket, nodes, par = make()
    plan = dlib.Plan(bucket)
    assert ring(plan) == (4, 4)
    C = nodes.shape[0]
    co = coeffs_for(bucket, plan.info, C)
    out = plan.assemble(_dev(nodes), _dev(par), _dev(co))
    torch.cuda.synchronize()
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert (got["info"] == 0).all()
    check_against_truth(oracle_mod, bucket, nodes, par, co, got, oracle_mod.OraclePlan(bucket).assemble(nodes, par, co))

"""Small buckets with at most as many cells as SMs: every cell has an SM to itself, so the calls take 16 warps
per cell (8, two CTAs per SM, with more), and the outputs of every entry point are the same bit for bit
on both sides of that line: the phases and their sums do not depend on the warps."""
import ctypes as ct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from camellia2_b200 import lib as dlib  # noqa: E402
from tests.helpers import cdr2d, coeffs_for, poisson2d, poisson3d, poisson_tri, stokes2d, stokes_tri  # noqa: E402

pytestmark = pytest.mark.gpu

ASSEMBLE, ADJOINT, ENERGY, DLS = range(4)


def shape(plan, kind, C):
    """(warps per CTA, CTAs per SM, CTAs per cell) of a call."""
    out = (ct.c_int * 5)()
    assert dlib.load().dpg_debug_launch_shape(plan.h, kind, C, out) == 0
    return tuple(out[:3])


def _dev(x):
    return None if x is None else torch.as_tensor(np.ascontiguousarray(x)).cuda()


# 4, 5, 9, 9, 8, 13, 10 and 12 test tiles; 3, 4, 5, 5, 6, 8, 7 and 5 trial tiles
@pytest.mark.parametrize("make", [lambda: poisson2d(1, 1), lambda: poisson_tri(2, 2), lambda: poisson2d(2, 2),
                                  lambda: poisson3d(1, 1), lambda: poisson_tri(3, 2), lambda: cdr2d(3, 2),
                                  lambda: stokes_tri(2, 1), lambda: stokes2d(1, 2)])
def test_few_cells_take_16_warps_and_give_the_same_bits(make):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _, bucket, nodes, par = make()
    plan = dlib.Plan(bucket)
    for kind in (ASSEMBLE, ENERGY, DLS):
        assert shape(plan, kind, 1) == shape(plan, kind, sms) == (16, 1, 1)
        assert shape(plan, kind, sms + 1) == (8, 2, 1)
    C, M = sms + 1, plan.info["M"]
    idx = np.arange(C) % nodes.shape[0]
    many = (_dev(nodes[idx]), _dev(par[idx]), _dev(coeffs_for(bucket, plan.info, C, seed=3)))
    g = torch.Generator(device="cuda").manual_seed(1)
    x, Kb, lb = (torch.randn(s, generator=g, dtype=torch.float64, device="cuda") for s in ((C, M), (C, M, M), (C, M)))
    few = tuple(None if t is None else t[:sms] for t in many)

    def calls(cells, n):
        out = list(plan.assemble(*cells).values()) + list(plan.parts(*cells)) + list(plan.dls(*cells))
        out += list(plan.energy_error(*cells, x[:n]))
        if cells[2] is not None:
            out += list(plan.adjoint(*cells, Kb[:n], lb[:n]))
        torch.cuda.synchronize()
        return out

    for a, b in zip(calls(few, sms), calls(many, C)):
        assert torch.equal(a, b[:sms])

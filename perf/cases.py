"""Timed workloads of the per-cell DPG assembly library, through its public Python entry points.

A case names an entry point ("op"), a formulation on one cell topology with its degrees (k, dk),
the number of cells C and the inverse cell size 1/h.  Cells are jittered squares, cubes or right
triangles of edge h at random places of the unit square or cube with random side parities: a
cell's outputs depend on its neighbours through the parities alone.  Cell sizes stay where the
FP64 Gram factorisation keeps ten digits of K and S.

The second half of the file computes the same outputs in plain torch float64: Legendre and
Dubiner test bases (K, S and the energy do not depend on the choice of test basis), one dense
product per matrix, torch's Cholesky, and torch's autograd for the reverse mode.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from camellia2_b200 import abi, formulation as fm, lib

QUAD, HEX, TRI = "quad", "hex", "tri"
TOPO = {QUAD: abi.TOPO_QUAD, HEX: abi.TOPO_HEX, TRI: abi.TOPO_TRI}
F64 = dict(dtype=torch.float64)


# ----------------------------------------------------------------------------
# The cases
# ----------------------------------------------------------------------------


def listed():
    def case(name, op, form, topo, k, dk, cells, inv_h):
        return dict(name=name, op=op, form=form, topo=topo, k=k, dk=dk, cells=cells, inv_h=inv_h)

    return [
        # the textbook 16 x 16 mesh: a call so small that latency decides
        case("poisson_quad_k2_16x16", "assemble", "poisson", QUAD, 2, 2, 256, 16),
        # the eight children of one refined hex, re-assembled after an adaptive step
        case("poisson_hex_k2_8", "assemble", "poisson", HEX, 2, 1, 8, 16),
        # a high-order production mesh in 2D
        case("poisson_quad_k4_128x128", "assemble", "poisson", QUAD, 4, 2, 16384, 16),
        # a nonlinear or inverse problem: one forward and one reverse sweep over a 128 x 128 mesh
        case("cdr_quad_k3_128x128", "assemble", "cdr", QUAD, 3, 2, 16384, 64),
        case("cdr_quad_k3_adjoint_128x128", "adjoint", "cdr", QUAD, 3, 2, 16384, 32),
        # an hp mesh of quads and triangles, p = 1..6, re-assembled as one graph every step
        case("stokes_forest_graph", "graph", "stokes", "mixed", 6, 2, 6000, 4),
        # the few cells that were raised to p = 6 after an adaptive step
        case("stokes_quad_p6_37", "assemble", "stokes", QUAD, 6, 2, 37, 8),
        # the 48^3 hex mesh, the largest call
        case("poisson_hex_k2_48cubed", "assemble", "poisson", HEX, 2, 1, 110592, 48),
        # its error indicator on a coarser mesh, the field recovery after the global solve, and the
        # global assembly over a fixed mesh, repeated every time step
        case("poisson_hex_k2_energy_20cubed", "energy", "poisson", HEX, 2, 1, 8000, 20),
        case("poisson_hex_k2_recover_40cubed", "recover", "poisson", HEX, 2, 1, 64000, 40),
        case("poisson_hex_k2_scatter_32cubed", "scatter", "poisson", HEX, 2, 1, 32768, 32),
        # host buffers in and out, as a CPU code that calls the library does
        case("poisson_hex_k2_host_17cubed", "host", "poisson", HEX, 2, 1, 4913, 17),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["assemble"] * 6 + ["adjoint", "graph", "energy", "recover", "scatter", "host"])
    if op == "graph":
        return dict(op=op, form="stokes", topo="mixed", k=rng.randint(2, 6), dk=2, cells=_log_int(rng, 200, 8000),
                    inv_h=rng.randint(2, 4))
    if op == "scatter":
        n = rng.randint(3, 34)
        return dict(op=op, form="poisson", topo=HEX, k=rng.randint(1, 2), dk=1, cells=n ** 3, inv_h=n)
    form, topo, k, dk = rng.choice([
        lambda: ("poisson", QUAD, rng.randint(1, 5), rng.randint(1, 2)),
        lambda: ("poisson", TRI, rng.randint(1, 5), 2),
        lambda: ("poisson", HEX, rng.choice([1, 2, 2, 3]), 1),
        lambda: ("cdr", QUAD, rng.randint(1, 4), rng.randint(1, 2)),
        lambda: ("stokes", QUAD, rng.randint(1, 6), 2),
        lambda: ("stokes", TRI, rng.randint(1, 6), 2),
    ])()
    if op == "adjoint":
        form, topo, k, dk = "cdr", QUAD, rng.randint(1, 3), rng.randint(1, 2)
    if op == "recover" and form == "stokes":  # the field blocks that the recovery takes
        k = min(k, 4)
    c = dict(op=op, form=form, topo=topo, k=k, dk=dk)
    # no dearer than the largest listed case
    z = _sizes(c)
    most = min(2.0 ** 16, 48.0 ** 3 * (282.0 / (z["N"] + z["M"])) ** 3 / (1 if op in ("assemble", "recover") else 8))
    c["cells"] = _log_int(rng, 1, max(2.0, most))
    c["inv_h"] = rng.randint(4, 16 if k >= 4 else 32)
    return c


def _form(name, dim):
    return {"poisson": lambda: fm.PoissonFormulation(dim), "cdr": lambda: fm.ConvectionDiffusionReactionFormulation(2),
            "stokes": lambda: fm.StokesVGPFormulation(2)}[name]()


def _plan(c):
    return lib.Plan(_form(c["form"], 3 if c["topo"] == HEX else 2).bucket(TOPO[c["topo"]], c["k"], c["dk"]))


CORNERS = {
    QUAD: [[0, 0], [1, 0], [1, 1], [0, 1]],
    TRI: [[0, 0], [1, 0], [0, 1]],
    HEX: [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]],
}
SIDES = {
    QUAD: [[0, 1], [1, 2], [2, 3], [3, 0]],
    TRI: [[0, 1], [1, 2], [2, 0]],
    HEX: [[0, 1, 5, 4], [1, 2, 6, 5], [2, 3, 7, 6], [0, 4, 7, 3], [0, 3, 2, 1], [4, 5, 6, 7]],
}


def _cells(c, gen, dev, levels=0):
    """Vertices (C, nv, d), parities (C, ns) and coefficients (C, slots, points)."""
    C, topo = c["cells"], c["topo"]
    corners = torch.tensor(CORNERS[topo], device=dev, **F64)
    d = corners.shape[1]
    n = torch.full((C, 1), float(c["inv_h"]), device=dev, **F64)
    if levels:  # refinement levels 0..levels, each half as likely as the one before
        u = torch.rand((C, 1), generator=gen, device=dev, **F64)
        n = n * torch.exp2(torch.clamp(torch.floor(-torch.log2(1.0 - u)), max=levels))
    at = torch.floor(torch.rand((C, d), generator=gen, device=dev, **F64) * n) / n
    nodes = at[:, None] + corners / n[:, None]
    nodes = nodes + (torch.rand(nodes.shape, generator=gen, device=dev, **F64) - 0.5) * 0.2 / n[:, None]
    parity = (torch.randint(0, 2, (C, len(SIDES[topo])), generator=gen, device=dev) * 2 - 1).to(torch.int8)
    z = _sizes(c)
    shape = (C, z["slots"], z["points"])
    if c["form"] != "cdr":  # loads
        return nodes, parity, torch.rand(shape, generator=gen, device=dev, **F64) * 2 - 1
    co = torch.empty(shape, device=dev, **F64)
    co[:, 0] = torch.exp(0.5 * (torch.randn((C, shape[2]), generator=gen, device=dev, **F64) - 4.0))  # sqrt(eps)
    theta = torch.rand((C, 1), generator=gen, device=dev, **F64) * (2 * math.pi)
    co[:, 1], co[:, 2] = torch.cos(theta), torch.sin(theta)
    co[:, 3] = torch.rand((C, shape[2]), generator=gen, device=dev, **F64)
    co[:, 4] = torch.rand((C, shape[2]), generator=gen, device=dev, **F64) * 2 - 1
    return nodes, parity, co


def _buckets(c):
    """The buckets of an hp mesh: 70 % quads, degrees 1..k equally likely."""
    out = []
    for topo, share in ((QUAD, 0.7), (TRI, 0.3)):
        for k in range(1, c["k"] + 1):
            out.append(dict(op="assemble", form=c["form"], topo=topo, k=k, dk=c["dk"], inv_h=c["inv_h"],
                            cells=max(1, round(c["cells"] * share / c["k"]) + (k * 7) % 5 - 2)))
    return out


def _trace_mesh(c, dev):
    """Local-to-global ids (C, t) of a conforming hex mesh's traces (H1 points identified by their
    lattice position, fluxes by face), the number of global dofs and the CSR graph."""
    n, k = c["inv_h"], c["k"]
    idx = torch.arange(n, device=dev)
    kk, jj, ii = torch.meshgrid(idx, idx, idx, indexing="ij")
    cell = torch.stack([ii.reshape(-1), jj.reshape(-1), kk.reshape(-1)], 1)
    P = k * n + 1
    bi, ai = torch.meshgrid(torch.arange(k + 1, device=dev), torch.arange(k + 1, device=dev), indexing="ij")
    ai, bi = ai.reshape(-1), bi.reshape(-1)
    h1, flux = [], []
    for face in range(6):
        a, side = face // 2, face % 2
        b, e = [x for x in range(3) if x != a]
        pos = [None] * 3
        pos[a] = (k * (cell[:, a] + side))[:, None].expand(-1, ai.numel())
        pos[b] = k * cell[:, b][:, None] + ai
        pos[e] = k * cell[:, e][:, None] + bi
        h1.append(pos[0] + P * (pos[1] + P * pos[2]))
        fid = a * (n + 1) * n * n + ((cell[:, a] + side) * n + cell[:, b]) * n + cell[:, e]
        flux.append(P ** 3 + fid[:, None] * k * k + torch.arange(k * k, device=dev))
    raw = torch.cat(h1 + flux, 1)
    uniq, gid = torch.unique(raw, return_inverse=True)
    ng = uniq.numel()
    key = torch.empty(0, dtype=torch.int64, device=dev)
    for g in torch.split(gid, 4096):  # the graph's (row, column) pairs
        key = torch.unique(torch.cat([key, torch.unique((g[:, :, None] * ng + g[:, None, :]).reshape(-1))]))
    row_ptr = torch.zeros(ng + 1, dtype=torch.int64, device=dev)
    row_ptr[1:] = torch.cumsum(torch.bincount(key // ng, minlength=ng), 0)
    return gid.contiguous(), ng, row_ptr, (key % ng).contiguous()


def _inputs(c, seed, dev):
    """The arrays a user's program has in hand before the call."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    rand = lambda *shape: torch.randn(shape, generator=gen, device=dev, **F64)  # noqa: E731
    z = _sizes(c) if c["op"] != "graph" else None
    C = c["cells"]
    if c["op"] == "graph":
        return dict(buckets=[_cells(b, gen, dev, levels=2) for b in _buckets(c)])
    if c["op"] == "recover":  # K of an SPD cell problem, the load, and the solved traces
        X = rand(C, z["M"], 24)
        K = torch.bmm(X, X.transpose(1, 2)).div_(24.0)
        K.diagonal(dim1=1, dim2=2).add_(0.5)
        return dict(K=K, l=rand(C, z["M"]), t=rand(C, z["t"]))
    if c["op"] == "scatter":
        S = rand(C, z["t"], z["t"])
        return dict(S=S + S.transpose(1, 2), s=rand(C, z["t"]))
    nodes, parity, coeff = _cells(c, gen, dev)
    st = dict(nodes=nodes, parity=parity, coeff=coeff)
    if c["op"] == "adjoint":  # J = sum_c r^T K r + g^T l
        r = rand(C, z["M"])
        st.update(Kbar=r[:, :, None] * r[:, None, :], lbar=rand(C, z["M"]))
    if c["op"] == "energy":
        st["x"] = rand(C, z["M"])
    return st


def prepare(case, seed):
    c, dev = case, torch.device("cuda")
    st = dict(_inputs(c, seed, dev), op=c["op"])
    if c["op"] == "graph":
        items = []
        for b, (nodes, parity, coeff) in zip(_buckets(c), st.pop("buckets")):
            plan = _plan(b)
            items.append((plan, nodes, parity, coeff, plan.alloc_outputs(b["cells"])))
        st["outs"] = [it[4] for it in items]
        st["graph"] = lib.Graph(items)
    elif c["op"] == "scatter":
        gid, ng, row_ptr, col = _trace_mesh(c, dev)
        C, t = gid.shape
        map_ptr = torch.arange(C * t + 1, dtype=torch.int64, device=dev)
        st["plan"] = lib.ScatterPlan(C, t, map_ptr, gid.reshape(-1), None, ng, row_ptr, col)
        st["values"] = torch.zeros(col.numel(), device=dev, **F64)
        st["rhs"] = torch.zeros(ng, device=dev, **F64)
    elif c["op"] == "host":
        plan = st["plan"] = _plan(c)
        for name in ("nodes", "parity", "coeff"):
            st[name] = st[name].cpu().pin_memory()
        st["out"] = {name: torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
                     for name, x in plan.alloc_outputs(c["cells"], "cpu").items()}
    else:
        st["plan"] = _plan(c)
        if c["op"] == "assemble":
            st["out"] = st["plan"].alloc_outputs(c["cells"])
    return st


def run(state):
    st = state
    op = st["op"]
    if op == "assemble":
        return st["plan"].assemble(st["nodes"], st["parity"], st["coeff"], out=st["out"])
    if op == "host":
        return st["plan"].assemble_host(st["nodes"], st["parity"], st["coeff"], out=st["out"])
    if op == "graph":
        st["graph"].launch()
        return st["outs"]
    if op == "adjoint":
        cbar, info = st["plan"].adjoint(st["nodes"], st["parity"], st["coeff"], st["Kbar"], st["lbar"])
        return dict(coeff_bar=cbar, info=info)
    if op == "energy":
        e, info = st["plan"].energy_error(st["nodes"], st["parity"], st["coeff"], st["x"])
        return dict(energy=e, info=info)
    if op == "recover":
        u, info = st["plan"].recover_fields(st["K"], st["l"], st["t"])
        return dict(u=u, info=info)
    st["values"].zero_()
    st["rhs"].zero_()
    st["plan"].apply(st["S"], st["s"], st["values"], st["rhs"])
    return dict(values=st["values"], rhs=st["rhs"])


def work(case):
    """Bytes: inputs and outputs once.  Operations: the lower triangle of G with four slots per point
    (value and gradient, or vector and divergence, fold every graph-norm term), B with its volume terms, the
    Cholesky factor of G, the triangular solve, K, and the condensation."""
    c = case
    if c["op"] == "graph":
        parts = [work(b) for b in _buckets(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    z, C = _sizes(c), c["cells"]
    N, M, t, f = z["N"], z["M"], z["t"], z["f"]
    nv, d = len(CORNERS[c["topo"]]), len(CORNERS[c["topo"]][0])
    if c["op"] == "recover":
        return dict(bytes=8.0 * C * (f * M + f + t + M) + 4 * C, flops=C * (f ** 3 / 3 + 2 * f * f + 2 * f * t))
    if c["op"] == "scatter":
        n, k = c["inv_h"], c["k"]
        dofs = 3 * n * n * (n + 1) * ((k - 1) ** 2 + k * k) + 3 * (k - 1) * n * (n + 1) ** 2 + (n + 1) ** 3
        local = 8 + 12 * (k - 1) + 6 * ((k - 1) ** 2 + k * k)  # distinct dofs of a cell
        face = 4 + 4 * (k - 1) + (k - 1) ** 2 + k * k
        nnz = C * local ** 2 - 3 * n * n * (n - 1) * face ** 2  # pairs shared by two cells counted once
        return dict(bytes=8.0 * (C * (t * t + t) + nnz + dofs + nnz), flops=float(C * (t * t + t)))
    inp = 8 * nv * d + len(SIDES[c["topo"]]) + 8 * z["slots"] * z["points"]
    out = 8 * (M * M + M + t * t + t) + 4
    form = 4.0 * z["QG"] * N * N + 8.0 * z["QB"] * N * f + N ** 3 / 3.0
    flops = form + N * N * (M + 1) + N * (M + 1) ** 2 + f ** 3 / 3.0 + f * f * (t + 1) + f * (t + 1) ** 2
    if c["op"] == "energy":
        inp, out, flops = inp + 8 * M, 12, form + N * N + 2 * N * M
    if c["op"] == "adjoint":
        inp, out = inp + 8 * (M * M + M), 8 * z["slots"] * z["points"] + 4
        # X = G^-1 [B F], P = X S_A, and the point products f^T X, f^T P of the pull-back
        flops = form + 2 * N * N * (M + 1) + 2.0 * N * (M + 1) ** 2 + 8.0 * (2 * z["QG"] + z["QB"]) * N * (M + 1)
    return dict(bytes=float(C) * (inp + out), flops=float(C) * flops)


# ----------------------------------------------------------------------------
# The same outputs in plain float64
# ----------------------------------------------------------------------------


def _gauss(n):
    return np.polynomial.legendre.leggauss(n)


def _gll(p):
    """Gauss-Lobatto nodes of degree p."""
    if p == 0:
        return np.zeros(1)
    inner = np.polynomial.legendre.Legendre.basis(p).deriv().roots() if p > 1 else np.zeros(0)
    return np.concatenate([[-1.0], np.sort(inner.real), [1.0]])


def _legendre(p, x):
    """Orthonormal Legendre values and derivatives (n, p + 1)."""
    L = [np.polynomial.legendre.Legendre.basis(i) * math.sqrt(i + 0.5) for i in range(p + 1)]
    return np.stack([b(x) for b in L], 1), np.stack([b.deriv()(x) for b in L], 1)


def _lagrange(nodes, x):
    """Values at x of the Lagrange functions of the 1D nodes."""
    p = len(nodes) - 1
    return np.linalg.solve(_legendre(p, nodes)[0].T, _legendre(p, np.asarray(x))[0].T).T


def _tensor_rule(d, degree):
    x, w = _gauss(degree // 2 + 1)
    grids = np.meshgrid(*([x] * d), indexing="ij")[::-1]  # x fastest
    ws = np.meshgrid(*([w] * d), indexing="ij")
    return np.stack([g.reshape(-1) for g in grids], 1), np.prod([u.reshape(-1) for u in ws], 0)


def _rule(topo, degree):
    if topo != TRI:
        return _tensor_rule(3 if topo == HEX else 2, degree)
    (xu, wu), (xv, wv) = _gauss(degree // 2 + 1), _gauss((degree + 1) // 2 + 1)
    v, u = [g.reshape(-1) for g in np.meshgrid(0.5 * (1 + xv), 0.5 * (1 + xu), indexing="ij")]
    b, a = [g.reshape(-1) for g in np.meshgrid(wv, wu, indexing="ij")]
    return np.stack([u * (1 - v), v], 1), 0.25 * a * b * (1 - v)


def _dubiner(p, x):
    """Polynomials of degree <= p on the unit triangle: values (n, m) and gradients (n, m, 2).
    phi_ij = P_i((2x + y - 1) / (1 - y)) (1 - y)^i P_j^(2i+1,0)(2y - 1), by recurrences without division."""
    X, Y = x[:, 0], x[:, 1]
    one, zero = np.ones_like(X), np.zeros_like(X)
    a, b = 2 * X + Y - 1, 1 - Y

    def mul(f, g):
        return f[0] * g[0], f[1] * g[0] + f[0] * g[1], f[2] * g[0] + f[0] * g[2]

    def lin(*terms):
        return tuple(sum(c * f[i] for c, f in terms) for i in range(3))

    A, B2, y1 = (a, 2 * one, one), mul((b, zero, -one), (b, zero, -one)), (2 * Y - 1, zero, 2 * one)
    Q = [(one, zero, zero), A]
    for i in range(1, p):
        Q.append(lin(((2 * i + 1) / (i + 1), mul(A, Q[i])), (-i / (i + 1), mul(B2, Q[i - 1]))))
    val, grad, deg = [], [], []
    for i in range(p + 1):
        al = 2.0 * i + 1
        J = [(one, zero, zero), lin(((al + 2) / 2, y1), (al / 2, (one, zero, zero)))]
        for j in range(1, p - i):
            m = j + 1
            a1 = 2 * m * (m + al) * (2 * m + al - 2)
            J.append(lin(((2 * m + al - 1) * (2 * m + al) * (2 * m + al - 2) / a1, mul(y1, J[j])),
                         ((2 * m + al - 1) * al * al / a1, J[j]),
                         (-2 * (m + al - 1) * (m - 1) * (2 * m + al) / a1, J[j - 1])))
        for j in range(p - i + 1):
            f = mul(Q[i], J[j])
            s = math.sqrt(2.0 * (2 * i + 1) * (i + j + 1))
            val.append(s * f[0])
            grad.append(np.stack([s * f[1], s * f[2]], 1))
            deg.append(i + j)
    return np.stack(val, 1), np.stack(grad, 1), np.array(deg)


def _scalar_test(topo, p, x):
    """Values (n, m) and reference gradients (n, m, d) of a basis of Q_p or P_p."""
    if topo == TRI:
        return _dubiner(p, x)[:2]
    d = x.shape[1]
    f = [_legendre(p, x[:, i]) for i in range(d)]

    def prod(deriv):
        out = np.ones((x.shape[0], 1))
        for i in reversed(range(d)):
            out = (out[:, :, None] * f[i][int(i == deriv)][:, None, :]).reshape(x.shape[0], -1)
        return out

    return prod(-1), np.stack([prod(i) for i in range(d)], 2)


def _vector_test(topo, n, x):
    """Values (n, m, d) and divergences (n, m) of a Raviart-Thomas basis of order n."""
    d = x.shape[1]
    val, div = [], []
    if topo == TRI:
        v, g, deg = _dubiner(n - 1, x)
        for c in range(2):
            e = np.zeros(v.shape + (2,))
            e[:, :, c] = v
            val.append(e)
            div.append(g[:, :, c])
        top = deg == n - 1
        val.append(v[:, top, None] * x[:, None, :])
        div.append(2 * v[:, top] + np.einsum("nmc,nc->nm", g[:, top], x))
        return np.concatenate(val, 1), np.concatenate(div, 1)
    for c in range(d):
        f = [_legendre(n if i == c else n - 1, x[:, i]) for i in range(d)]
        for out, deriv in ((val, -1), (div, c)):
            m = np.ones((x.shape[0], 1))
            for i in reversed(range(d)):
                m = (m[:, :, None] * f[i][int(i == deriv)][:, None, :]).reshape(x.shape[0], -1)
            if out is div:
                out.append(m)
            else:
                e = np.zeros(m.shape + (d,))
                e[:, :, c] = m
                out.append(e)
    return np.concatenate(val, 1), np.concatenate(div, 1)


def _tri_nodes(p):
    """Warp and blend points of degree p on the unit triangle, rows of constant y."""
    alpha = [0.0, 0.0, 1.4152, 0.1001, 0.2751, 0.98][p - 1]
    even, gll = np.linspace(-1, 1, p + 1), _gll(p)

    def warp(r):
        return (_lagrange(even, np.array([r])) @ (gll - even))[0] / (1 - r * r) if abs(r) < 1 - 1e-10 else 0.0

    out = []
    for n in range(p + 1):
        for m in range(p + 1 - n):
            l1, l3 = n / p, m / p
            l2 = 1 - l1 - l3
            x, y = l3 - l2, (2 * l1 - l2 - l3) / math.sqrt(3)
            for i, (u, v, o) in enumerate(((l2, l3, l1), (l3, l1, l2), (l1, l2, l3))):
                w = 4 * u * v * warp(v - u) * (1 + (alpha * o) ** 2)
                x += w * math.cos(2 * math.pi * i / 3)
                y += w * math.sin(2 * math.pi * i / 3)
            out.append([(3 * x - math.sqrt(3) * y + 2) / 6, (math.sqrt(3) * y + 1) / 3])
    return np.array(out)


def _field(topo, k, x):
    """Nodal basis of the L2 fields (degree k - 1) at x."""
    p = k - 1
    if p == 0:
        return np.ones((x.shape[0], 1))
    if topo == TRI:
        return np.linalg.solve(_dubiner(p, _tri_nodes(p))[0].T, _dubiner(p, x)[0].T).T
    out = np.ones((x.shape[0], 1))
    for i in reversed(range(x.shape[1])):
        out = (out[:, :, None] * _lagrange(_gll(p), x[:, i])[:, None, :]).reshape(x.shape[0], -1)
    return out


def _trace(p, x):
    """Nodal basis of degree p on a reference side."""
    out = np.ones((x.shape[0], 1))
    for i in reversed(range(x.shape[1])):
        out = (out[:, :, None] * _lagrange(_gll(p), x[:, i])[:, None, :]).reshape(x.shape[0], -1)
    return out


def _shape(topo, x):
    """Vertex shape functions (n, nv) and their derivatives (n, nv, d)."""
    if topo == TRI:
        N = np.stack([1 - x[:, 0] - x[:, 1], x[:, 0], x[:, 1]], 1)
        return N, np.broadcast_to(np.array([[-1.0, -1.0], [1.0, 0.0], [0.0, 1.0]]), (x.shape[0], 3, 2))
    v = 2.0 * np.array(CORNERS[topo]) - 1
    f = 0.5 * (1 + x[:, None, :] * v)
    N = f.prod(2)
    d = x.shape[1]
    dN = np.stack([0.5 * v[:, i] * np.prod([f[:, :, j] for j in range(d) if j != i], 0) for i in range(d)], 2)
    return N, dN


def _terms(form, d):
    """Bilinear form as data.  tests: g(rad) or d(iv) spaces; volume terms (field, test, operator,
    constant, slot); side terms (trace, test, operator, constant, slot, normal component);
    load terms (test, slot); traces: degree offset and whether the side parity multiplies them."""
    if form == "poisson":
        vol = [(0, 1, "div", 1.0, None)]
        vol += [(1 + i, 1, i, 1.0, None) for i in range(d)] + [(1 + i, 0, "d%d" % i, -1.0, None) for i in range(d)]
        side = [(0, 1, "n", -1.0, None, None), (1, 0, "v", 1.0, None, None)]
        return dict(tests="gd", nfields=1 + d, vol=vol, side=side, traces=[(0, False), (-1, True)], load=[(0, 0)], slots=1)
    if form == "cdr":
        vol = [(0, 1, "div", 1.0, 0), (0, 0, "v", 1.0, 3)]
        for i in range(2):
            vol += [(1 + i, 1, i, 1.0, None), (1 + i, 0, "d%d" % i, 1.0, 0), (0, 0, "d%d" % i, -1.0, 1 + i)]
        side = [(0, 1, "n", -1.0, 0, None), (1, 0, "v", -1.0, None, None)]
        return dict(tests="gd", nfields=3, vol=vol, side=side, traces=[(0, False), (-1, True)], load=[(0, 4)], slots=5)
    vol, side = [], []
    for i in range(2):
        vol += [(i, 2 + i, "div", 1.0, None), (2, i, "d%d" % i, -1.0, None), (i, 4, "d%d" % i, -1.0, None)]
        vol += [(3 + 2 * i + j, 2 + i, j, 1.0, None) for j in range(2)]
        vol += [(3 + 2 * i + j, i, "d%d" % j, 1.0, None) for j in range(2)]
        side += [(i, 2 + i, "n", -1.0, None, None), (2 + i, i, "v", 1.0, None, None), (i, 4, "v", 1.0, None, i)]
    return dict(tests="ggddg", nfields=7, vol=vol, side=side, traces=[(0, False)] * 2 + [(-1, True)] * 2,
                load=[(0, 0), (1, 1)], slots=2)


def _sizes(c):
    topo, k, r = c["topo"], c["k"], c["k"] + c["dk"]
    d = 3 if topo == HEX else 2
    T = _terms(c["form"], d)
    if topo == TRI:
        card = dict(g=(r + 1) * (r + 2) // 2, d=r * (r + 2))
        per_field = k * (k + 1) // 2
        rule = lambda n: (n // 2 + 1) * ((n + 1) // 2 + 1)  # noqa: E731
    else:
        card = dict(g=(r + 1) ** d, d=d * (r + 1) * r ** (d - 1))
        per_field = k ** d
        rule = lambda n: (n // 2 + 1) ** d  # noqa: E731
    f = T["nfields"] * per_field
    ns = len(SIDES[topo])
    t = sum(ns * (k + 1 + o) ** (d - 1) for o, _ in T["traces"])
    QG, QB, QS = rule(2 * r), rule(k + r), ((k + r) // 2 + 1) ** (d - 1)
    return dict(N=sum(card[s] for s in T["tests"]), M=f + t, f=f, t=t, QG=QG, QB=QB, QS=QS, slots=T["slots"],
                points=QG + QB + ns * QS)


class _Reference:
    """Dense float64 assembly of one bucket."""

    def __init__(self, c, dev):
        topo, k, r = c["topo"], c["k"], c["k"] + c["dk"]
        self.dev, self.topo, self.d = dev, topo, 3 if topo == HEX else 2
        self.T, self.z = _terms(c["form"], self.d), _sizes(c)
        up = lambda a: torch.tensor(np.ascontiguousarray(a), device=dev, **F64)  # noqa: E731

        def tables(x, w):
            p = dict(w=up(w), dN=up(_shape(topo, x)[1]), field=up(_field(topo, k, x)))
            p["g"], p["gg"] = [up(a) for a in _scalar_test(topo, r, x)]
            p["d"], p["dd"] = [up(a) for a in _vector_test(topo, r, x)]
            return p

        self.G, self.B = tables(*_rule(topo, 2 * r)), tables(*_rule(topo, k + r))
        xs, ws = _tensor_rule(self.d - 1, k + r)
        Ns, dNs = _shape(QUAD, xs) if self.d == 3 else (np.stack([0.5 * (1 - xs[:, 0]), 0.5 * (1 + xs[:, 0])], 1),
                                                       np.broadcast_to(np.array([[[-0.5], [0.5]]]), (len(xs), 2, 1)))
        v = np.array(CORNERS[topo], float) if topo == TRI else 2.0 * np.array(CORNERS[topo]) - 1
        self.sides = []
        for sv in SIDES[topo]:
            p = tables(Ns @ v[sv], ws)
            p["tang"] = up(np.einsum("na,xat->nxt", v[sv].T, dNs).transpose(1, 0, 2))  # (q, d, d - 1)
            self.sides.append(p)
        self.tr = [up(_trace(k + o, xs)) for o, _ in self.T["traces"]]

    def _geometry(self, p, nodes):
        J = torch.einsum("cai,qaj->cqij", nodes, p["dN"])
        return J, torch.linalg.det(J), torch.linalg.inv(J)

    def _op(self, p, geo, test, op):
        """Operator values (C, q, m) of a test var."""
        J, det, Ji = geo
        if self.T["tests"][test] == "g":
            if op == "v":
                return p["g"][None].expand(J.shape[0], -1, -1)
            return torch.einsum("cqj,qmj->cqm", Ji[:, :, :, int(op[1])], p["gg"])
        if op == "div":
            return p["dd"][None] / det[:, :, None]
        if op == "n":
            return torch.einsum("cqi,cqij,qmj->cqm", p["normal"], J / det[:, :, None, None], p["d"])
        return torch.einsum("cqj,qmj->cqm", J[:, :, op] / det[:, :, None], p["d"])

    def system(self, nodes, parity, coeff):
        """G (C, N, N), B (C, N, M) and F (C, N)."""
        T, z, d, C = self.T, self.z, self.d, nodes.shape[0]
        m = [(self.G["g"] if s == "g" else self.G["dd"]).shape[1] for s in T["tests"]]
        off = np.concatenate([[0], np.cumsum(m)])
        geo = self._geometry(self.G, nodes)
        rows = [[(t, op, co, sl) for f, t, op, co, sl in T["vol"] if f == i] for i in range(T["nfields"])]
        for t, s in enumerate(T["tests"]):  # the L2 part of the graph norm
            rows += [[(t, "v", 1.0, None)]] if s == "g" else [[(t, i, 1.0, None)] for i in range(d)]
        Lr = []
        for row in rows:
            L = torch.zeros((C, z["QG"], off[-1]), device=self.dev, **F64)
            for t, op, co, sl in row:
                v = co * self._op(self.G, geo, t, op)
                if sl is not None:
                    v = v * coeff[:, sl, :z["QG"], None]
                L = L + torch.nn.functional.pad(v, (int(off[t]), int(off[-1] - off[t + 1])))
            Lr.append(L * torch.sqrt(self.G["w"] * geo[1])[:, :, None])
        L = torch.cat(Lr, 1)
        G = L.transpose(1, 2) @ L
        # B: blocks (test var) x (trial var), and F
        nf = self.B["field"].shape[1]
        cols = [nf] * T["nfields"] + [len(SIDES[self.topo]) * x.shape[1] for x in self.tr]
        blocks = [[0.0] * len(cols) for _ in m]
        F = [torch.zeros((C, n), device=self.dev, **F64) for n in m]
        geo = self._geometry(self.B, nodes)
        wd = self.B["w"] * geo[1]
        pts = slice(z["QG"], z["QG"] + z["QB"])
        for f, t, op, co, sl in T["vol"]:
            s = co * wd if sl is None else co * wd * coeff[:, sl, pts]
            blocks[t][f] = blocks[t][f] + (self._op(self.B, geo, t, op) * s[:, :, None]).transpose(1, 2) @ self.B["field"]
        for t, sl in T["load"]:
            F[t] = F[t] + torch.einsum("cqm,cq->cm", self._op(self.B, geo, t, "v"), wd * coeff[:, sl, pts])
        per_side = {}
        for i, p in enumerate(self.sides):
            geo = self._geometry(p, nodes)
            tg = torch.einsum("cqij,qjt->cqit", geo[0], p["tang"])
            n = (torch.stack([tg[:, :, 1, 0], -tg[:, :, 0, 0]], 2) if d == 2
                 else torch.linalg.cross(tg[..., 0], tg[..., 1], dim=2))
            meas = n.norm(dim=2)
            p = dict(p, normal=n / meas[:, :, None])
            pts = slice(z["QG"] + z["QB"] + i * z["QS"], z["QG"] + z["QB"] + (i + 1) * z["QS"])
            for b, t, op, co, sl, nc in T["side"]:
                s = co * p["w"] * meas
                s = s if sl is None else s * coeff[:, sl, pts]
                s = s if nc is None else s * p["normal"][:, :, nc]
                s = s * parity[:, i:i + 1].double() if T["traces"][b][1] else s
                v = (self._op(p, geo, t, op) * s[:, :, None]).transpose(1, 2) @ self.tr[b]
                per_side.setdefault((t, b), {}).setdefault(i, []).append(v)
        for (t, b), by_side in per_side.items():
            blocks[t][T["nfields"] + b] = torch.cat([sum(by_side[i]) for i in range(len(self.sides))], 2)
        zero = lambda t, j: torch.zeros((C, m[t], cols[j]), device=self.dev, **F64)  # noqa: E731
        B = torch.cat([torch.cat([x if torch.is_tensor(x) else zero(t, j) for j, x in enumerate(row)], 2)
                       for t, row in enumerate(blocks)], 1)
        return G, B, torch.cat(F, 1)

    def whitened(self, nodes, parity, coeff):
        """W = L^-1 B and y = L^-1 F, G = L L^T."""
        G, B, F = self.system(nodes, parity, coeff)
        s = torch.rsqrt(G.diagonal(dim1=1, dim2=2))
        L = torch.linalg.cholesky(G * s[:, :, None] * s[:, None, :])
        W = torch.linalg.solve_triangular(L, torch.cat([B, F[:, :, None]], 2) * s[:, :, None], upper=False)
        return W[:, :, :-1], W[:, :, -1]

    def outputs(self, nodes, parity, coeff):
        W, y = self.whitened(nodes, parity, coeff)
        K = W.transpose(1, 2) @ W
        l = torch.einsum("cnm,cn->cm", W, y)
        f = self.z["f"]
        X = torch.cholesky_solve(torch.cat([K[:, :f, f:], l[:, :f, None]], 2), torch.linalg.cholesky(K[:, :f, :f]))
        S = K[:, f:, f:] - K[:, f:, :f] @ X[:, :, :-1]
        s = l[:, f:] - (K[:, f:, :f] @ X[:, :, -1:])[:, :, 0]
        return dict(K=K, l=l, S=S, s=s, info=None)


def _chunks(c, arrays, fn):
    """fn over slices of the cells, its results joined."""
    z = _sizes(c)
    n = max(1, int(2.0e9 / (8.0 * z["N"] * (24 * z["QG"] + 2 * z["N"] + 2 * z["M"]))))
    parts = [fn(*[a[i:i + n] for a in arrays]) for i in range(0, c["cells"], n)]
    return {k: (None if parts[0][k] is None else torch.cat([p[k] for p in parts])) for k in parts[0]}


def exact(case, seed):
    c = case
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    st = _inputs(c, seed, dev)
    if c["op"] == "recover":
        z = _sizes(c)
        f = z["f"]
        rhs = st["l"][:, :f] - (st["K"][:, :f, f:] @ st["t"][:, :, None])[:, :, 0]
        u = torch.linalg.solve(st["K"][:, :f, :f], rhs)
        return dict(u=torch.cat([u, st["t"]], 1), info=None)
    if c["op"] == "scatter":
        gid, ng, row_ptr, col = _trace_mesh(c, dev)
        key = torch.repeat_interleave(torch.arange(ng, device=dev), row_ptr.diff()) * ng + col
        values = torch.zeros(col.numel(), device=dev, **F64)
        rhs = torch.zeros(ng, device=dev, **F64).index_add_(0, gid.reshape(-1), st["s"].reshape(-1))
        for g, S in zip(torch.split(gid, 4096), torch.split(st["S"], 4096)):
            at = torch.searchsorted(key, (g[:, :, None] * ng + g[:, None, :]).reshape(-1))
            values.index_add_(0, at, S.reshape(-1))
        return dict(values=values, rhs=rhs)
    if c["op"] == "graph":
        return [_chunks(b, a, _Reference(b, dev).outputs) for b, a in zip(_buckets(c), st["buckets"])]
    R = _Reference(c, dev)
    cells = [st["nodes"], st["parity"], st["coeff"]]
    if c["op"] == "energy":
        def energy(nodes, parity, coeff, x):
            W, y = R.whitened(nodes, parity, coeff)
            return dict(energy=(y - (W @ x[:, :, None])[:, :, 0]).norm(dim=1), info=None)

        return _chunks(c, cells + [st["x"]], energy)
    if c["op"] == "adjoint":
        def adjoint(nodes, parity, coeff, Kbar, lbar):
            coeff = coeff.clone().requires_grad_(True)
            W, y = R.whitened(nodes, parity, coeff)
            J = (W.transpose(1, 2) @ W * Kbar).sum() + (torch.einsum("cnm,cn->cm", W, y) * lbar).sum()
            return dict(coeff_bar=torch.autograd.grad(J, coeff)[0], info=None)

        return _chunks(c, cells + [st["Kbar"], st["lbar"]], adjoint)
    out = _chunks(c, cells, R.outputs)
    return {k: (v if v is None or c["op"] != "host" else v.cpu()) for k, v in out.items()}

"""The count of vertex values read (algorithmic_values), restated for passes that end at the first level.

A tolerance that every first test meets leaves five nodes per Simpson subdomain and the two boundary nodes
of every task, at positions that follow from the meshes alone.  A vertex read at (w, v, v') takes two mesh
points per argument strictly between mesh points, one per argument on a mesh point or beyond a fermionic
mesh, and none beyond the bosonic one (buffer.jl:51-84); the arguments are those of flow_su2_{s,t,u}.jl.
"""
import math
from bisect import bisect_left

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def arguments(X, slot, W, v, F):
    """Arguments of the s, t and u channel of one vertex of bubble X (F: its fermionic task frequency)."""
    h = 0.5
    if X == 0:
        if slot == 0:
            return ((W, F, -v), (v - F, h * (W + v + F), h * (W - v - F)), (v + F, h * (W - v + F), h * (W + v - F)))
        return ((W, v, F), (-v - F, h * (W + v - F), h * (W - v + F)), (v - F, h * (W + v + F), h * (W - v - F)))
    if X == 1:
        if slot == 0:
            return ((v + F, h * (-W - v + F), h * (-W + v - F)), (W, F, v), (-v + F, h * (-W + v + F), h * (W + v + F)))
        if slot == 1:
            return ((v + F, h * (-W + v - F), h * (-W - v + F)), (W, v, F), (v - F, h * (-W + v + F), h * (W + v + F)))
        if slot == 2:
            return ((v + F, h * (W + v - F), h * (-W + v - F)), (-v + F, h * (W + v + F), h * (-W + v + F)), (W, v, F))
        return ((v + F, h * (W - v + F), h * (-W - v + F)), (v - F, h * (W + v + F), h * (-W + v + F)), (W, F, v))
    if slot == 0:
        return ((v + F, h * (W - v + F), h * (-W - v + F)), (v - F, h * (W + v + F), h * (-W + v + F)), (W, F, v))
    return ((v + F, h * (W + v - F), h * (-W + v - F)), (-v + F, h * (W + v + F), h * (-W + v + F)), (W, v, F))


def points(x, mesh):
    """Mesh points that interpolation at |x| <= mesh[-1] reads."""
    x = abs(x)
    return 1 if mesh[bisect_left(mesh, x)] == x else 2


def corners(args, Om, nu):
    w, v, vp = args
    if abs(w) > Om[-1]:
        return 0
    n = points(w, Om)
    for f in (v, vp):
        if abs(f) <= nu[-1]:
            n *= points(f, nu)
    return n


def expected(m, Ns, rows, C, Lam):
    """(nodes, values) of a one-loop pass at eval = 1, all subdomains ending at their first test."""
    nodes = values = 0
    S, T = (m.omega_s.tolist(), m.nu_s.tolist()), (m.omega_t.tolist(), m.nu_t.tolist())
    for X in range(3):
        Om, nu = T if X == 1 else S
        val = Om[-1] + nu[-1]
        inf = math.inf
        pairs = [(inf, inf)] + [(f, inf) for f in nu] + [(inf, g) for g in nu]
        pairs += [(f, g) for k, g in enumerate(nu) for f in nu[k:]]
        tasks = [(W, f, g) for W in Om for f, g in pairs]
        for W, f, g in tasks:
            a = 2.0 * (Lam + 0.5 * W)
            xs = [-val, val]
            ranges = [(-a, 0.0, 1.0), (0.0, a, 1.0)]
            if val > a:
                b = math.pow(val / a, 1.0) * a
                ranges += [(a, b, -1.0), (a, b, 1.0)]
            for lo, hi, sg in ranges:
                h = 0.5 * (hi - lo) / 2.0
                xs += [sg * lo, sg * (lo + h), sg * (0.5 * (lo + hi)), sg * (lo + 3.0 * h), sg * hi]
            for v in xs:
                n = 0
                for slot in range(4 if X == 1 else 2):
                    c = sum(corners(q, *(T if ch == 1 else S))
                            for ch, q in enumerate(arguments(X, slot, W, v, g if slot & 1 else f)))
                    n += c * (Ns if slot < 2 else 1)
                values += C * (n + 3 * Ns + (2 * rows if X == 1 else 0))
            nodes += len(xs)
    return nodes, values


@pytest.mark.parametrize("lattice, size, model, J, symmetry", [
    ("square", 3, "heisenberg", [[1.0]], "su2"),
    ("kagome", 2, "kagome-xxz-dm", [[1.0, 0.8, 0.2]], "u1-dm"),
])
def test_values_of_a_first_level_pass(pkg, lattice, size, model, J, symmetry):
    import pffrg_gb300.workloads as wl
    from pffrg_gb300.flow import FlowContext

    w = wl.Workload("t", lattice, size, model, J, 1, 1.0, 9, 3, 2, 0.02, 3, symmetry=symmetry)
    lat, r, m, a = wl.build_state(w)
    da = pkg.action.Action.empty_like(a)
    with FlowContext(r, m, symmetry=symmetry, precision="fp64") as ctx:
        ctx.compute_dgamma(1.0, a, da, 1, (1e12, 1.0))
        st = ctx.read_stats()
    nodes, values = expected(m, r.num_sites, sum(len(o) for o in r.overlap), 2 if symmetry == "su2" else 6, 1.0)
    assert np.isfinite(da.buf).all()
    assert st["integrand_evals"] == nodes
    assert st["algorithmic_values"] == values

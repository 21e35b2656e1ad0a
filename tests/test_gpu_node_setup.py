"""Propagators and interpolation plans of the passes where they switch form, FP64 against the oracle.

Λ = 0.05 takes exp(-w²/Λ²) below 2^-1022 on most of the mesh (and w beyond the last σ point), Λ = 20
keeps it near one, where G needs exp - 1; every task reads its own channel at mesh frequencies, whose
plans hold two corners of eight.  The bound is that of the other FP64 parity tests: adaptive decisions
and nodes are the oracle's, so only the rounding of a node differs (1e-10 of the largest entry).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lam", [0.05, 0.4, 20.0])
@pytest.mark.parametrize("lattice, size, model, J, symmetry", [
    ("square", 3, "heisenberg", [[1.0]], "su2"),
    ("kagome", 2, "kagome-xxz-dm", [[1.0, 0.8, 0.2]], "u1-dm"),
])
def test_fp64_rhs_matches_oracle(pkg, O, lattice, size, model, J, symmetry, Lam):
    import pffrg_gb300.workloads as wl
    from pffrg_gb300.flow import FlowContext

    w = wl.Workload("t", lattice, size, model, J, 1, Lam, 11, 4, 3, 0.02, 3, symmetry=symmetry)
    lat, r, m, a = wl.build_state(w)
    P = O.Problem(r, m, symmetry=symmetry) if symmetry != "su2" else O.Problem(r, m)
    ref = np.zeros_like(a.buf)
    O.dsigma(P, Lam, a.buf, ref)
    O.dgamma(P, 1, Lam, a.buf, ref, 3)
    da = pkg.action.Action.empty_like(a)
    with FlowContext(r, m, symmetry=symmetry, precision="fp64") as ctx:
        ctx.compute_dsigma(Lam, a, da)
        ctx.compute_dgamma(Lam, a, da, 3)
    assert np.max(np.abs(da.buf - ref)) < 1e-10 * np.max(np.abs(ref))

"""FP64 propagators at cutoffs so small that the constants of the regulator leave the range of a double.

Λ = 1e-105: 2/Λ³ overflows while exp(-w²/Λ²) is zero at every frequency, so the single-scale propagator
and with it dΓ are exactly zero.  Λ = 1e-153: w²/Λ² overflows from w = 14 on, where exp(-w²/Λ²) is zero
and G = 1/(w + Σ).  A tolerance that every first test meets keeps the 1/w² integrands of that cutoff to
five nodes per subdomain; with the nodes fixed only their rounding differs from the oracle's, 1e-10 of the
largest entry as in the other FP64 parity tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODELS = [("square", 3, "heisenberg", [[1.0]], "su2"), ("kagome", 2, "kagome-xxz-dm", [[1.0, 0.8, 0.2]], "u1-dm")]


def problem(O, lattice, size, model, J, symmetry):
    import pffrg_gb300.workloads as wl

    w = wl.Workload("t", lattice, size, model, J, 1, 1.0, 11, 4, 3, 0.02, 3, symmetry=symmetry)
    lat, r, m, a = wl.build_state(w)
    return r, m, a, O.Problem(r, m, symmetry=symmetry) if symmetry != "su2" else O.Problem(r, m)


@pytest.mark.parametrize("lattice, size, model, J, symmetry", MODELS)
def test_katanin_bubbles_vanish_below_the_range_of_the_exponential(pkg, O, lattice, size, model, J, symmetry):
    from pffrg_gb300.flow import FlowContext

    Lam = 1e-105
    r, m, a, P = problem(O, lattice, size, model, J, symmetry)
    ref = np.zeros_like(a.buf)
    O.dsigma(P, Lam, a.buf, ref)
    O.dgamma(P, 1, Lam, a.buf, ref, 3)
    assert not ref.any()
    da = pkg.action.Action.empty_like(a)
    with FlowContext(r, m, symmetry=symmetry, precision="fp64") as ctx:
        ctx.compute_dsigma(Lam, a, da)
        ctx.compute_dgamma(Lam, a, da, 3)
    assert not da.buf.any()


@pytest.mark.parametrize("lattice, size, model, J, symmetry", MODELS)
def test_plain_bubbles_where_the_exponent_overflows(pkg, O, lattice, size, model, J, symmetry):
    from pffrg_gb300.flow import FlowContext

    Lam, tol = 1e-153, (1e12, 1.0)
    r, m, a, P = problem(O, lattice, size, model, J, symmetry)
    ref = np.zeros_like(a.buf)
    corrs = O.sde(P, Lam, a.buf, ref, 2, tol, tol)
    O.bse(P, Lam, a.buf, ref, corrs, 2, tol)
    got = pkg.action.Action.empty_like(a)
    with FlowContext(r, m, symmetry=symmetry, precision="fp64") as ctx:
        ctx.compute_sigma_sde(Lam, a, got, 2, tol, tol)
        ctx.compute_gamma_bse(Lam, a, got, 2, tol)
    assert np.isfinite(ref).all() and np.max(np.abs(ref)) > 0
    assert np.max(np.abs(got.buf - ref)) < 1e-10 * np.max(np.abs(ref))

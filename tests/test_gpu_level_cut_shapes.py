"""Fine and coarse cuts of a level on lattices whose lanes hold one, two and three sites.

A chunk capacity just above what the coarse cut needs forbids most finer cuts, provided that the largest level
has few chunks per subdomain: small meshes and a tolerance of 2 %, which a jump of the integrand meets after
some six levels.  That the two runs were cut differently shows in the last bits of the FP64 sums.  Bounds: FP64 2^12 terms x 2^-53 < 1e-12 of the largest
entry; mixed: the hand-off to FP64 agrees up to the FP32 rounding of its bound, so that a subdomain at its edge
may keep the FP32 rounding 2^-24 of its values, 1e-7 of the largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lattice, size, model, J, symmetry", [
    ("square", 5, "heisenberg", [[1.0]], "su2"),                      # 12 sites: 16 lanes
    ("diamond", 7, "heisenberg", [[1.0]], "su2"),                     # 35 sites: two per lane
    ("kagome", 8, "kagome-xxz-dm", [[1.0, 0.8, 0.2]], "u1-dm"),       # 82 sites: three per lane
])
def test_cuts_agree(pkg, lattice, size, model, J, symmetry, precision):
    import pffrg_gb300._capi as C
    import pffrg_gb300.workloads as wl
    from pffrg_gb300.flow import FlowContext

    w = wl.Workload("t", lattice, size, model, J, 1, 1.0, 9, 3, 2, 0.1, 5, symmetry=symmetry)
    lat, r, m, a = wl.build_state(w)

    def rhs(ctx):
        da = pkg.action.Action.empty_like(a)
        ctx.compute_dsigma(1.0, a, da)
        ctx.compute_dgamma(1.0, a, da, 1, (1e-6, 2e-2))
        return ctx.last_integrand_evals, da.buf.copy()

    with FlowContext(r, m, symmetry=symmetry, precision=precision) as ctx:
        nodes, fine = rhs(ctx)
        refused, cap = 64, 1 << 17
        coarse = None
        while cap - refused > refused // 16:
            mid = (cap + refused) // 2
            ctx.set_capacities(queue_chunks=mid)
            try:
                n, coarse = rhs(ctx)
                cap = mid
            except C.PffrgError as e:
                assert e.code == C.PFFRG_E_LIMIT, str(e)
                refused = mid
    assert coarse is not None and refused > 64
    top = np.max(np.abs(fine))
    if precision == "fp64":
        assert n == nodes
        assert not np.array_equal(fine, coarse), "both runs used the same cut"
    assert np.max(np.abs(coarse - fine)) <= (1e-12 if precision == "fp64" else 1e-7) * top

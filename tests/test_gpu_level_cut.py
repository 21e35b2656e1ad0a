"""How a level of the adaptive quadrature is cut into chunks does not change its result.

Levels with few active subdomains are cut finer than 32 nodes per chunk, as far as half the chunk
capacity allows; a capacity just large enough for the coarse cut therefore forbids most of the fine
ones.  Both must evaluate the same nodes and give the same sums up to the order in which a
subdomain's chunk sums are added: FP64 2^12 terms x 2^-53 < 1e-12, FP32 chunks with compensated sums
(second-order error, 4096 terms x 2^-48) < 1e-10 of the largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def symmetry(model):
    return "u1-dm" if model == "kagome-xxz-dm" else "su2"


def state(lattice, size, model, J):
    import pffrg_gb300.workloads as wl

    return wl.build_state(wl.Workload("t", lattice, size, model, J, 1, 1.0, 11, 4, 3, 0.1, 5, symmetry=symmetry(model)))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lattice, size, model, J", [
    ("square", 3, "heisenberg", [[1.0]]),            # 6 sites: 8 lanes, one node per batch
    ("square", 5, "heisenberg", [[1.0]]),            # 12 sites: 16 lanes, two nodes
    ("honeycomb", 7, "heisenberg", [[1.0]]),         # 18 sites: 32 lanes, four nodes
    ("kagome", 3, "kagome-xxz-dm", [[1.0, 0.8, 0.2]]),
])
def test_fine_and_coarse_cuts_agree(pkg, lattice, size, model, J, precision):
    import pffrg_gb300._capi as C
    from pffrg_gb300.flow import FlowContext

    lat, r, m, a = state(lattice, size, model, J)
    got = []
    with FlowContext(r, m, symmetry=symmetry(model), precision=precision) as ctx:
        ctx.upload(C.SLOT_A, a)

        def rhs():
            ctx.rhs(1.0, 2)
            da = pkg.action.Action.empty_like(a)
            ctx.download(C.SLOT_DA, da)
            got.append((ctx.last_integrand_evals, da.buf.copy()))

        for waves in (True, False):
            ctx.set_async_waves(waves)
            ctx.set_capacities()
            rhs()
            cap = 64
            while True:
                ctx.set_capacities(queue_chunks=cap)
                try:
                    rhs()
                    break
                except C.PffrgError as e:
                    assert e.code == C.PFFRG_E_LIMIT, str(e)
                    cap *= 2
            assert cap > 64, "no capacity refused: the state does not reach the chunk limit"
    tol = 1e-12 if precision == "fp64" else 1e-10
    for n, buf in got[1:]:
        assert n == got[0][0]
        assert np.max(np.abs(buf - got[0][1])) <= tol * np.max(np.abs(got[0][1]))

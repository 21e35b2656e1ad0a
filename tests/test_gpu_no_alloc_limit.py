"""Which problems the no-allocation entry point takes: its byte count, restated.

A caller that sizes its problems by the limit finds the same ones accepted from version to version, so
the count keeps 56 bytes per subdomain and two lists of 16-byte chunk records whatever the passes hold.
Square L = 3 with 19 bosonic and 12 fermionic frequencies at eval 10 lies 1.9 MB beyond the array with
that count (and 1.9 MB within it without the records' last 16 bytes); at eval 9 it fits.
"""
import re

import pytest

import test_zz_no_alloc as base

pytestmark = pytest.mark.gpu


def counted_bytes(Ns, rows, nsig, NO, Nn, eval_):
    up = lambda x: (x + 255) & ~255  # noqa: E731
    tasks = NO * (1 + 2 * Nn + Nn * (Nn + 1) // 2)
    nsub = tasks * 3 * (4 * eval_ + 1)
    queue = 2 * nsub + 4096
    vec = 16 * Ns
    blocks = [4 * Ns, 4 * (Ns + 1), 4 * rows, 16 * (nsig + 2 * NO + 2 * Nn), 16 * NO * (eval_ + 1), 16 * tasks, 48 * NO,
              32 * 2048 * 6 * NO, 4]  # tables, meshes, log bounds, tasks, corrections, Gauss-Kronrod segments, flag
    blocks += [56 * nsub, vec * nsub, vec * nsub, 16 * queue, 16 * queue, 4 * nsub, 4 * nsub, vec * queue, 8 * queue,
               4 * nsub, 32]
    return sum(map(up, blocks))


@pytest.mark.parametrize("eval_, fits", [(10, False), (9, True)])
def test_limit_of_the_no_allocation_entry(pkg, eval_, fits):
    import torch

    import pffrg_gb300.workloads as wl

    lib = base._lib()
    w = wl.Workload("noalloc", "square", 3, "heisenberg", [[1.0]], 1, 1.0, 11, 18, 11, 0.02, 3)
    lat, r, m, a = wl.build_state(w)
    need = counted_bytes(r.num_sites, sum(len(o) for o in r.overlap), len(m.sigma), len(m.omega_s), len(m.nu_s), eval_)
    assert (need <= lib.pffrg_noalloc_scratch_bytes()) == fits
    a_dev = torch.from_numpy(a.buf.copy()).cuda()
    da_dev = torch.zeros_like(a_dev)
    rc = base._call(lib, r, m, a, a_dev, da_dev, 1.0, eval_, (1e6, 1.0))
    msg = lib.pffrg_noalloc_last_error().decode()
    if fits:
        assert rc == 0, msg
    else:
        assert rc == base.LIMIT, (rc, msg)
        assert int(re.search(r"needs (\d+) bytes", msg).group(1)) == need
        assert float(da_dev.abs().max()) == 0.0  # nothing was written

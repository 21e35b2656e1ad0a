"""Performance cases of the flow library: what a flow, a parquet solve and their measurements call.

Every case is one call (or the few calls that belong together) through the public Python entry points,
on a seeded state of a lattice model:

* ``rhs``: one flow right-hand side with host arrays in and out (compute_dsigma, then compute_dgamma);
* ``step``: one Bogacki-Shampine step on the device and the download of the new state, what ``launch``
  does per step when it writes files or calls back;
* ``chi``: the static correlations of a state, measured after every accepted step;
* ``parquet``: iterations of the parquet fixed point that a flow starts from;
* ``resample``: the mesh cuts and the move of the state onto the next meshes after an accepted step.

States: ``flow`` is smooth in every frequency, peaked on the scale of the cutoff and decaying over the
sites, as vertices along a flow are; ``noise`` is independent normal noise on every entry (the benchmark
workloads' states), whose integrands have a jump or a kink at every mesh point and refine deepest.
"""
from __future__ import annotations

import importlib
import math

import numpy as np

import __graft_entry__

__graft_entry__.load_package()
_action = importlib.import_module("pffrg_gb300.action")
_capi = importlib.import_module("pffrg_gb300._capi")
_flow = importlib.import_module("pffrg_gb300.flow")
_freq = importlib.import_module("pffrg_gb300.frequency")
_lattice = importlib.import_module("pffrg_gb300.lattice")
_workloads = importlib.import_module("pffrg_gb300.workloads")


def _case(name, op, lattice, size, mesh, Lam, *, model="heisenberg", J="1.0", loops=1, precision="fp64", state="flow",
          noise=0.05, eval_=None, sigma_corr=False, num_chi=0, iters=0):
    c = {"op": op, "lattice": lattice, "size": size, "model": model, "J": J, "num_sigma": mesh[0],
         "num_omega": mesh[1], "num_nu": mesh[2], "Lam": Lam, "loops": loops, "precision": precision, "state": state,
         "noise": noise, "eval": eval_ or _flow.get_eval(Lam, 10, 100), "sigma_corr": sigma_corr,
         "num_chi": num_chi, "iters": iters}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a trial run's lattice and meshes, few tasks, latency and launches count
        _case("rhs-square3-small-fp64", "rhs", "square", 3, (11, 4, 3), 1.0, eval_=2),
        # the first configuration a user meets (square L = 3, one loop, default meshes) along a flow
        _case("rhs-square3-1l-mixed", "rhs", "square", 3, (50, 15, 10), 1.0, precision="mixed"),
        # the same lattice on a noisy state in FP64: few sites, deep refinement everywhere
        _case("rhs-square3-1l-fp64-noise", "rhs", "square", 3, (50, 15, 10), 1.0, state="noise", noise=0.1),
        # the benchmark: pyrochlore L = 6 (48 sites, 8047 overlap rows), two loops, noisy state
        _case("rhs-pyrochlore6-2l-mixed", "rhs", "pyrochlore", 6, (50, 15, 10), 1.0, loops=2, precision="mixed",
              state="noise"),
        # the comparator's precision on the same lattice along a flow
        _case("rhs-pyrochlore6-1l-fp64", "rhs", "pyrochlore", 6, (25, 10, 7), 0.8),
        # U(1)-DM, six components, many sites, three loops with the self-energy corrections
        _case("rhs-kagome8-dm-3l-mixed", "rhs", "kagome", 8, (20, 8, 6), 1.0, model="kagome-xxz-dm", J="1.0,0.8,0.2",
              loops=3, precision="mixed", sigma_corr=True),
        # U(1)-DM on a small lattice in FP64, odd mesh sizes
        _case("rhs-kagome3-dm-1l-fp64", "rhs", "kagome", 3, (17, 9, 5), 2.5, model="kagome-xxz-dm", J="1.0,0.8,0.2"),
        # one step of a two-loop flow in its middle, the work that a flow repeats
        _case("step-honeycomb5-2l-mixed", "step", "honeycomb", 5, (25, 15, 10), 1.5, loops=2, precision="mixed"),
        # one step at a small cutoff, where the integration ranges are cut finest
        _case("step-cubic4-1l-mixed-low", "step", "cubic", 4, (25, 12, 8), 0.12, precision="mixed"),
        # correlations of a state in the upper half of a flow on the default χ mesh
        _case("chi-square4-fp64", "chi", "square", 4, (25, 15, 10), 4.0, num_chi=10),
        # the parquet start of a flow (a few of its iterations)
        _case("parquet-honeycomb4-fp64", "parquet", "honeycomb", 4, (25, 15, 10), 2.0, iters=3),
        # onto the next meshes after an accepted step, the largest default state
        _case("resample-pyrochlore6", "resample", "pyrochlore", 6, (50, 15, 10), 1.0),
    ]


# lattices and sizes that draws choose from, with the sites and overlap rows they reduce to
_DRAW_SU2 = [("square", 3, 6, 55), ("square", 4, 9, 136), ("square", 5, 12, 286), ("square", 6, 16, 541),
             ("square", 8, 25, 1531), ("honeycomb", 3, 5, 38), ("honeycomb", 5, 11, 218), ("honeycomb", 7, 18, 716),
             ("kagome", 4, 13, 299), ("kagome", 6, 26, 1327), ("kagome", 7, 34, 2300), ("triangular", 5, 12, 426),
             ("triangular", 7, 20, 1424), ("cubic", 3, 7, 74), ("cubic", 5, 16, 658), ("cubic", 6, 23, 1581),
             ("diamond", 5, 15, 605), ("diamond", 7, 35, 4423), ("pyrochlore", 4, 18, 885),
             ("pyrochlore", 5, 31, 3007), ("pyrochlore", 6, 48, 8047)]
_DRAW_DM = [("kagome", 2, 7, 47), ("kagome", 3, 14, 218), ("kagome", 4, 23, 591), ("kagome", 5, 34, 1321),
            ("kagome", 6, 48, 2641), ("kagome", 8, 82, 7772)]


def _tasks(c):
    """Channel tasks of one pass with v >= v' (3 channels)."""
    no, nn = c["num_omega"] + 1, c["num_nu"] + 1
    return 3 * no * (1 + 2 * nn + nn * (nn + 1) // 2)


def _draw_cost(c, sites, rows):
    """Vertex operations of the first quadrature level, weighted by how deep the state refines and by what the
    precision costs: a measure to keep draws below the largest listed case."""
    comps = 6 if c["model"] == "kagome-xxz-dm" else 2
    nodes = _tasks(c) * (4 * c["eval"] + 1) * 5
    per_node = comps * sites * 60 + 2 * comps * rows / 3
    passes = {1: 1, 2: 3, 3: 6}[c["loops"]] * {"rhs": 1, "step": 4}.get(c["op"], 1)
    if c["op"] == "parquet":
        passes = 2 * c["iters"]
    deep = (4 if c["state"] == "flow" else 14) * (5 if c["precision"] == "fp64" else 1)
    return nodes * per_node * passes * deep


def draw(rng):
    logu = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    while True:
        op = rng.choices(["rhs", "step", "chi", "parquet", "resample"], [8, 4, 2, 2, 1])[0]
        dm = op in ("rhs", "step") and rng.random() < 0.3
        lat, size, sites, rows = rng.choice(_DRAW_DM if dm else _DRAW_SU2)
        mesh = (round(logu(11, 50)), round(logu(4, 16)), round(logu(3, 11)))
        Lam = round(logu(0.12, 8.0), 4)
        loops = rng.choice([1, 1, 2, 3]) if op in ("rhs", "step") else 1
        state = "noise" if op == "rhs" and rng.random() < 0.3 else "flow"
        if op == "chi":
            Lam = round(logu(3.0, 8.0), 4)
            if sites > 12:
                continue
        c = _case(None, op, lat, size, mesh, Lam, model="kagome-xxz-dm" if dm else "heisenberg",
                  J="1.0,%.3f,%.3f" % (rng.uniform(0.3, 1.2), rng.uniform(0.05, 0.4)) if dm else "1.0", loops=loops,
                  precision=rng.choice(["fp64", "mixed"]) if op in ("rhs", "step") else "fp64", state=state,
                  noise=round(logu(0.02, 0.1), 4), sigma_corr=loops == 3 and rng.random() < 0.5,
                  num_chi=rng.randint(5, 13) if op == "chi" else 0, iters=rng.randint(1, 3) if op == "parquet" else 0)
        if _draw_cost(c, sites, rows) < 4e11:
            return c


# ---------------------------------------------------------------------------
_models: dict = {}


def _model(case):
    """Lattice and its symmetry reduction, which a program builds once per model."""
    key = (case["lattice"], case["size"], case["model"], case["J"])
    if key not in _models:
        J, _ = _workloads.normalize_couplings([[float(x) for x in case["J"].split(",")]])
        lat = _lattice.get_lattice(case["lattice"], case["size"])
        _models[key] = lat, _lattice.get_reduced_lattice(case["model"], J, lat)
    return _models[key]


def _smooth(a, m, Lam, rng):
    """Vertices as along a flow: sums of Lorentzians in every frequency with widths around Λ that differ from site to
    site, on a background that reaches the asymptotic kernels continuously; amplitudes decay over the sites."""
    ns = a.layout.num_sites
    for v in a.Γ:
        for ch, (Om, nu) in zip(v.channels, ((m.omega_s, m.nu_s), (m.omega_t, m.nu_t), (m.omega_s, m.nu_s))):
            for q in (ch.q1, ch.q2_1, ch.q2_2, ch.q3):
                q[...] = 0.0
            for scale in (0.12, 0.04):
                amp = rng.normal(0.0, scale, ns) / (1.0 + 0.3 * np.arange(ns))
                f = amp[:, None] / (1.0 + (Om[None, :] / (rng.uniform(0.8, 3.0, (ns, 1)) * Lam)) ** 2)
                h = rng.uniform(-0.8, 1.5, (ns, 1)) / (1.0 + (nu[None, :] / (rng.uniform(0.7, 2.5, (ns, 1)) * Lam)) ** 2)
                ch.q1[...] += f
                ch.q2_1[...] += f[:, :, None] * (1.0 + h)[:, None, :]
                ch.q2_2[...] += f[:, :, None] * (1.0 + h)[:, None, :]
                ch.q3[...] += (f[:, :, None] * (1.0 + h)[:, None, :])[:, :, :, None] * (1.0 + h)[:, None, None, :]
    s = m.sigma
    a.Σ[...] = rng.uniform(0.1, 0.4) * s * Lam / (s * s + Lam * Lam)


def _state(case, seed):
    """(reduced lattice, meshes, action) of a case."""
    lat, r = _model(case)
    m = _freq.initial_mesh(case["Lam"], case["num_sigma"], case["num_omega"], case["num_nu"], case["num_chi"] or 10)
    a = _action.get_action_empty(_symmetry(case), r, m)
    if case["op"] == "parquet":
        # the couplings themselves start a parquet solve; another seed is another strength
        _action.init_action(lat, r, a)
        k = 1.0 + 0.3 * np.random.default_rng(seed).uniform(-1.0, 1.0)
        for v in a.Γ:
            v.bare *= k
        return r, m, a
    if case["state"] == "noise":
        _workloads.fill_noise(a, case["noise"], seed)
    else:
        _smooth(a, m, case["Lam"], np.random.default_rng(seed))
    _action.init_action(lat, r, a)
    return r, m, a


def _symmetry(case):
    return "u1-dm" if case["model"] == "kagome-xxz-dm" else "su2"


def _next_mesh(case):
    return _freq.initial_mesh(0.93 * case["Lam"], case["num_sigma"], case["num_omega"], case["num_nu"], 10)


def prepare(case, seed):
    r, m, a = _state(case, seed)
    ctx = _flow.FlowContext(r, m, symmetry=_symmetry(case), precision=case["precision"])
    s = {"case": case, "ctx": ctx, "m": m, "a": a, "out": _action.Action.empty_like(a)}
    if case["op"] == "step":
        ctx.upload(_capi.SLOT_A, a)
    elif case["op"] == "resample":
        ctx.upload(_capi.SLOT_NEXT, a)
        s["next"] = _next_mesh(case)
    return s


def run(s):
    c, ctx, a, out = s["case"], s["ctx"], s["a"], s["out"]
    if c["op"] == "rhs":
        ctx.compute_dsigma(c["Lam"], a, out)
        ctx.compute_dgamma(c["Lam"], a, out, c["eval"], loops=c["loops"], sigma_corr=c["sigma_corr"])
        return _parts(out)
    if c["op"] == "step":
        err, amax = ctx.bs_step(c["Lam"], 0.05 * c["Lam"], c["eval"], loops=c["loops"], sigma_corr=c["sigma_corr"])
        ctx.download(_capi.SLOT_NEXT, out)
        return dict(_parts(out), err=err, abs_max=amax)
    if c["op"] == "chi":
        return {"chi": ctx.compute_chi(c["Lam"], a, s["m"].chi)}
    if c["op"] == "parquet":
        ctx.upload(_capi.SLOT_A, a)
        it, abs_err, rel_err, hist = ctx.parquet(c["Lam"], c["eval"], max_iter=c["iters"], parquet_tol=(1e-12, 1e-12),
                                                 history=True)
        ctx.download(_capi.SLOT_A, out)
        return dict(_parts(out), iterations=it, residuals=hist)
    ctx.set_mesh(s["m"])
    sig, arg, cuts = ctx.scan_cuts(_capi.SLOT_NEXT)
    ctx.resample(_capi.SLOT_NEXT, _capi.SLOT_A, s["next"])
    ctx.download(_capi.SLOT_A, out)
    return dict(_parts(out), scan_sigma=sig, scan_argmax=arg, scan_cuts=cuts)


def _parts(a):
    """Self energy and vertex of an action, as the caller's arrays hold them."""
    n = a.layout.num_sigma
    return {"sigma": a.buf[:n], "vertex": a.buf[n:]}


def work(case):
    """Bytes: the state read and the result written once.  Operations: the bubbles of every task on the nodes that
    each Simpson subdomain needs for its first test (four new ones and the two corrections at the ends); how much
    deeper a state refines is not known before the call."""
    _, r = _model(case)
    comps = 6 if _symmetry(case) == "u1-dm" else 2
    no, nn, ns = case["num_omega"] + 1, case["num_nu"] + 1, r.num_sites
    size = case["num_sigma"] + 1 + comps * (ns + 3 * ns * no * (1 + nn) ** 2)
    if case["op"] == "resample":
        return {"bytes": 16 * size, "flops": 16 * size}
    if case["op"] == "chi":
        # nine boxes of the (v, v') plane, one 17-point rule each, on every site and frequency
        return {"bytes": 8 * size, "flops": 9 * 17 * (case["num_chi"] + 1) * ns * 100}
    rows = sum(len(o) for o in r.overlap)
    nodes = _tasks(case) / 3 * (16 * case["eval"] + 2)
    bubbles = nodes * comps * (3 * 6 * ns + 3 * rows)  # s, u: six operations a site; t: also the overlap rows
    passes = {1: 1, 2: 2.5, 3: 5}[case["loops"]]
    if case["op"] == "step":
        passes *= 4
    elif case["op"] == "parquet":
        passes = case["iters"]
    return {"bytes": 16 * size, "flops": bubbles * passes}


# ---------------------------------------------------------------------------
def _weights(x, mesh):
    """Interval and weights of linear interpolation on an increasing mesh, constant beyond its end."""
    hi = np.clip(np.searchsorted(mesh, x, side="left"), 1, len(mesh) - 1)
    t = np.clip((x - mesh[hi - 1]) / (mesh[hi] - mesh[hi - 1]), 0.0, 1.0)
    W = np.zeros((len(x), len(mesh)))
    W[np.arange(len(x)), hi - 1] = 1.0 - t
    W[np.arange(len(x)), hi] += t
    return W


def exact(case, seed):
    """Resampling in plain numpy.  The adaptive integrals have no such value here: what they return is fixed by
    the decisions of their refinement, subdomain by subdomain (10^4 to 10^5 of them, with up to 10^4 nodes each,
    and the bisections of the correction and self-energy integrals one after another), which plain array code
    does not follow in the time there is for it."""
    if case["op"] != "resample":
        return None
    r, m, a = _state(case, seed)
    n = _next_mesh(case)
    lay = a.layout
    res = np.zeros_like(a.buf)
    # Σ is odd in the frequency and falls off as 1/σ beyond its mesh
    inside = n.sigma <= m.sigma[-1]
    res[:lay.num_sigma] = np.where(inside, _weights(n.sigma, m.sigma) @ a.Σ, m.sigma[-1] * a.Σ[-1] / np.maximum(n.sigma, 1e-300))
    res[0] = 0.0
    shape = (lay.num_sites, lay.num_omega, lay.num_nu, lay.num_nu)
    cuts, arg = [], []
    for c, v in enumerate(a.Γ):
        res[lay.bare_offset(c):lay.bare_offset(c) + lay.num_sites] = v.bare
        for ch, (q, Om, nu, Om1, nu1) in enumerate(zip(v.channels, (m.omega_s, m.omega_t, m.omega_s), (m.nu_s, m.nu_t, m.nu_s),
                                                       (n.omega_s, n.omega_t, n.omega_s), (n.nu_s, n.nu_t, n.nu_s))):
            WO, WN = _weights(Om1, Om), _weights(nu1, nu)
            new = (np.einsum("xa,sa->sx", WO, q.q1), np.einsum("xa,yb,sab->sxy", WO, WN, q.q2_1, optimize=True),
                   np.einsum("xa,yb,sab->sxy", WO, WN, q.q2_2, optimize=True),
                   np.einsum("xa,yb,zc,sabc->sxyz", WO, WN, WN, q.q3, optimize=True))
            for k, x in enumerate(new):
                o = lay.kernel_offset(c, ch, k)
                res[o:o + x.size] = x.reshape(-1, order="F")
            top = int(np.argmax(np.abs(q.q3).reshape(-1, order="F")))
            s, w, i, j = np.unravel_index(top, shape, order="F")
            k = np.arange(lay.num_nu)
            arg.append(top)
            cuts.append(np.concatenate([q.q3[s, :, i, j], q.q3[s, w, k, k] - q.q3[s, w, -1, -1],
                                        q.q3[s, w, :, j] - q.q3[s, w, -1, j], q.q3[s, w, i, :] - q.q3[s, w, i, -1]]))
    return {"sigma": res[:lay.num_sigma], "vertex": res[lay.num_sigma:], "scan_sigma": a.Σ.copy(),
            "scan_argmax": np.array(arg, dtype=np.int64), "scan_cuts": np.array(cuts)}

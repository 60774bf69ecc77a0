"""The work that programs built on hiten_gb300 have it do, as timed cases.

Each case is one call of a public entry point at the sizes of the package's
own workloads (`hiten_gb300.workloads`, `bench.py`, the reference services'
defaults) or odd sizes between them.  Kinds:

* ``orbit``     one or a few trajectories with dense samples (a single
                `propagate` of the reference): latency.
* ``fixed``     fixed-step Runge-Kutta, 6-dim states or 42-dim state + STM.
* ``stability`` monodromy matrices of K periodic orbits (adaptive, 42-dim,
                each orbit its own period, last dense sample).
* ``manifold``  manifold seeds to the plane x = 1 - mu (terminal event),
                one call or a batch prepared once.
* ``section``   Poincare section of a synodic map: up to `hits` crossings.
* ``correct``   halo correction (Newton + Armijo) as one graph.
* ``detect``    crossings on already-sampled trajectories (SynodicMap.compute).
* ``filters``   acceptance filters of Manifold.compute on sampled trajectories.
* ``pairs``     the searches of find_connections between two section clouds.
"""
import math

import numpy as np
import torch

from hiten_gb300 import connections, corrector, halo, manifold, propagate, synodic, workloads

MU = workloads.MU_EM
DEV = "cuda"


def listed():
    return [
        # one halo orbit with 1000 samples: the reference's orbit.propagate(), the smallest call
        {"name": "orbit_1", "kind": "orbit", "n": 1, "m": 1000, "tf": 2.75},
        # fixed-step RK4 of a ragged set of states backward in time, every row kept (a trajectory plot)
        {"name": "rk4_777", "kind": "fixed", "order": 4, "dim": 6, "n": 777, "steps": 500, "every": 1, "fwd": -1},
        # state + STM by fixed-step RK8, the workload of workloads.stm_fixed_batch
        {"name": "rk8_stm_1024", "kind": "fixed", "order": 8, "dim": 42, "n": 1024, "steps": 3000, "every": 1000,
         "fwd": 1},
        # monodromy matrices of an odd number of orbits (stability.compute_stability)
        {"name": "stability_97", "kind": "stability", "n": 97},
        # an unstable manifold's seeds, odd count, below the scheduled driver's threshold
        {"name": "manifold_1237", "kind": "manifold", "n": 1237, "tf": 6.5, "forward": 1, "prepared": False},
        # the headline: the stable manifold's 512 x 32 seeds through a prepared batch
        {"name": "manifold_16384", "kind": "manifold", "n": 16384, "tf": 8.0, "forward": -1, "prepared": True},
        # a full synodic section map: 65536 states, up to 8 crossings each
        {"name": "section_65536", "kind": "section", "n": 65536, "tf": 20.0, "hits": 8},
        # a handful of halo corrections (one family's members), latency
        {"name": "correct_33", "kind": "correct", "n": 33},
        # a catalogue of halo corrections
        {"name": "correct_2048", "kind": "correct", "n": 2048},
        # crossings found on sampled trajectories, cubic interpolation, ragged count
        {"name": "detect_20011", "kind": "detect", "n": 20011, "m": 301, "interp": "cubic", "direction": -1},
        # acceptance filters of a manifold of 50 phases x 32 displacements at the service's default sampling
        {"name": "filters_1600", "kind": "filters", "n": 1600, "m": 4713},
        # connections between two sections of 65536 points: both radius pairings, both nearest-neighbour scans
        {"name": "pairs_65536", "kind": "pairs", "n": 65536, "n2": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["orbit", "fixed", "fixed", "stability", "manifold", "section", "correct", "detect", "filters",
                       "pairs"])
    if kind == "orbit":
        return {"kind": kind, "n": _log(rng, 1, 16), "m": _log(rng, 100, 2000), "tf": round(rng.uniform(0.5, 2.75), 3)}
    if kind == "fixed":
        dim = rng.choice([6, 42])
        n = _log(rng, 1, 4096 if dim == 42 else 16384)
        steps = _log(rng, 100, 3000 if n <= 1024 else 600)
        return {"kind": kind, "order": rng.choice([4, 6, 8]), "dim": dim, "n": n, "steps": steps,
                "every": max(1, steps // rng.randint(2, 8)), "fwd": rng.choice([1, -1])}
    if kind == "stability":
        return {"kind": kind, "n": _log(rng, 1, 2048)}
    if kind == "manifold":
        return {"kind": kind, "n": _log(rng, 50, 16384), "tf": round(rng.uniform(4.0, 8.0), 3),
                "forward": rng.choice([1, -1]), "prepared": rng.choice([True, False])}
    if kind == "section":
        return {"kind": kind, "n": _log(rng, 64, 65536), "tf": round(rng.uniform(3.0, 20.0), 3),
                "hits": rng.choice([1, 2, 4, 8])}
    if kind == "correct":
        return {"kind": kind, "n": _log(rng, 1, 2048)}
    if kind == "detect":
        return {"kind": kind, "n": _log(rng, 16, 65536), "m": _log(rng, 51, 301),
                "interp": rng.choice(["linear", "cubic"]), "direction": rng.choice([-1, 0, 1])}
    if kind == "filters":
        n = _log(rng, 50, 16384)
        return {"kind": kind, "n": n, "m": _log(rng, 100, 4713 if n <= 1600 else 500)}
    return {"kind": kind, "n": _log(rng, 200, 65536), "n2": _log(rng, 200, 65536)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _orbit_states(n, seed):
    """Halo-like states near L1 (the ranges of workloads.stm_fixed_batch)."""
    return workloads.stm_fixed_batch(n, seed=seed)[:, 36:].copy()


def _halo_guesses(n, seed):
    point, az, zen = workloads.halo_guess_params(n, seed=seed)
    out = np.empty((n, 6))
    for p in (1, 2):
        k = point == p
        if k.any():
            out[k] = halo.third_order_guess(MU, p, az[k], zen[k])
    return out


def _stability_inputs(n, seed):
    """Third-order halo orbits, each with a period of its own."""
    rng = np.random.default_rng(seed)
    return workloads.identity_stm_state(_halo_guesses(n, seed)), rng.uniform(1.5, 2.8, n)


def _manifold_seeds(n, forward, seed):
    """n seeds: as many phases as n // 32, log-uniform displacements."""
    stable = forward < 0
    n_disp = 32 if n >= 1024 else 8
    n_phase = -(-n // n_disp)
    t, phi = manifold.stm_grid(workloads.HALO_L1_AZ02_X0, workloads.HALO_L1_AZ02_T, MU, forward=forward)
    v = manifold.stable_eigvec(phi[-1, :36].reshape(6, 6), stable=stable)
    fr, di = workloads.manifold_grid(n_phase, n_disp, seed=seed)
    return manifold.seeds(t, phi, workloads.HALO_L1_AZ02_T, fr, di, v)[:n]


def _clouds(n, n2, seed):
    """Noisy closed curves on the (y, vy) plane, as manifold cuts look."""
    rng = np.random.default_rng(seed)

    def curve(k, phase):
        s = rng.uniform(0, 1, k)
        return np.c_[0.1 * np.cos(2 * np.pi * s + phase) + rng.normal(0, 1e-4, k),
                     0.3 * np.sin(2 * np.pi * s + phase) + rng.normal(0, 1e-4, k)]

    return curve(n, 0.0), curve(n2, 0.3)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = {"case": case}
    if kind == "orbit":
        s["y0"] = _dev(_orbit_states(n, seed))
    elif kind == "fixed":
        y = workloads.stm_fixed_batch(n, seed=seed)
        s["y0"] = _dev(y if case["dim"] == 42 else y[:, 36:])
        s["t"] = np.linspace(0.0, case["steps"] * 1e-3, case["steps"] + 1)
    elif kind == "stability":
        y, T = _stability_inputs(n, seed)
        s["y0"], s["T"] = _dev(y), T
    elif kind == "manifold":
        s["y0"] = _dev(_manifold_seeds(n, case["forward"], seed))
        if case["prepared"]:
            ev = propagate.EventSpec(index=0, offset=1.0 - MU, direction=0, max_hits=1)
            s["batch"] = propagate.Dop853Batch(n, 6, 0.0, case["tf"], MU, fwd=case["forward"], flip=(0, 6), event=ev)
    elif kind == "section":
        s["y0"] = _dev(workloads.section_states(n, seed=seed))
    elif kind == "correct":
        s["guess"] = _halo_guesses(n, seed)
    elif kind == "detect":
        s["t"] = torch.linspace(0.0, 3.0, case["m"], dtype=torch.float64, device=DEV)
        s["samples"] = propagate.propagate_dop853(_dev(workloads.section_states(n, seed=seed)), 0.0, 3.0, MU,
                                                  rtol=1e-11, atol=1e-11, max_steps=3000,
                                                  n_samples=case["m"]).samples
    elif kind == "filters":
        s["samples"] = propagate.propagate_dop853(_dev(_manifold_seeds(n, 1, seed)), 0.0, 1.5 * np.pi, MU,
                                                  max_steps=3000, n_samples=case["m"]).samples
    else:
        s["pu"], s["ps"] = (_dev(a) for a in _clouds(n, case["n2"], seed))
        s["matcher"] = connections.GpuSectionMatcher()
        s["coord"] = float(max(s["pu"].abs().max(), s["ps"].abs().max()))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _result(r):
    return {k: v for k, v in vars(r).items() if v is not None}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "orbit":
        return _result(propagate.propagate_dop853(state["y0"], 0.0, case["tf"], MU, n_samples=case["m"]))
    if kind == "fixed":
        rows, status = propagate.propagate_fixed(state["y0"], state["t"], MU, order=case["order"],
                                                 out_every=case["every"], fwd=case["fwd"], return_status=True)
        return {"rows": rows, "status": status}
    if kind == "stability":
        return _result(propagate.propagate_dop853(state["y0"], 0.0, state["T"], MU, n_samples=2000,
                                                  sample_last_only=True))
    if kind == "manifold":
        if case["prepared"]:
            return _result(state["batch"].run(state["y0"]))
        return _result(manifold.propagate_to_plane(state["y0"], MU, tf=case["tf"], forward=case["forward"]))
    if kind == "section":
        return _result(synodic.integrate_and_detect(state["y0"], MU, tf=case["tf"], max_hits=case["hits"]))
    if kind == "correct":
        r = corrector.correct_halo_graph(state["guess"], MU)
        return {"x0": r.x0, "half_period": r.half_period, "iterations": r.iterations,
                "residual_norm": r.residual_norm, "status": r.status}
    if kind == "detect":
        t, y, n = synodic.detect(state["t"], state["samples"], section_axis="y", plane_coords=("x", "vx"),
                                 direction=case["direction"], interp=case["interp"], max_hits=8)
        return {"hit_t": t, "hit_y": y, "n_hits": n}
    if kind == "filters":
        return manifold.trajectory_filters(state["samples"], MU)
    m, pu, ps, c = state["matcher"], state["pu"], state["ps"], state["coord"]
    return {"us": m.radius_best(pu, ps, 1e-4, c), "su": m.radius_best(ps, pu, 1e-4, c),
            "u": m.nearest(pu, c), "s": m.nearest(ps, c)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _stages(dim, stages, pairs):
    """Operations of one Runge-Kutta step: right-hand sides and stage sums
    (quotient, root and power count as one operation)."""
    rhs = 31 if dim == 6 else 31 + 60 + 6 * 18
    return stages * rhs + 2 * pairs * dim


def work(case):
    kind, n = case["kind"], case["n"]
    # DOP853: 12 right-hand sides, 58 stage products, 16 error products, the norm
    dop = {d: _stages(d, 12, 58 + 16) + 9 * d for d in (6, 42)}
    if kind == "orbit":  # about 10 accepted steps per unit of time
        return {"bytes": 8.0 * n * (6 + 6 * case["m"]), "flops": n * (10.0 * case["tf"] * dop[6] + 84.0 * case["m"])}
    if kind == "fixed":
        s, p = {4: (4, 7), 6: (7, 23), 8: (13, 70)}[case["order"]]
        rows = case["steps"] // case["every"] + 1
        return {"bytes": 8.0 * n * case["dim"] * (1 + rows),
                "flops": float(n) * case["steps"] * _stages(case["dim"], s, p)}
    if kind == "stability":
        return {"bytes": 8.0 * n * 42 * 3, "flops": n * 17.0 * dop[42]}
    if kind == "manifold":  # about 7 accepted steps per unit of time
        return {"bytes": 8.0 * n * 6 * 3, "flops": n * 7.0 * case["tf"] * dop[6]}
    if kind == "section":  # about 12 accepted steps per unit of time
        return {"bytes": 8.0 * n * 6 * (2 + case["hits"]), "flops": n * 12.0 * case["tf"] * dop[6]}
    if kind == "correct":  # about 6 Newton iterations: an event leg and an STM leg of 28 steps each
        return {"bytes": 8.0 * n * 6 * 2, "flops": n * 6.0 * 28.0 * (dop[6] + dop[42])}
    if kind == "detect":  # the section function's value at every sample, one candidate segment's scan per hit
        return {"bytes": 8.0 * n * case["m"], "flops": n * (8.0 * case["m"] + 51 * 20.0)}
    if kind == "filters":
        return {"bytes": 48.0 * n * case["m"], "flops": 40.0 * n * case["m"]}
    n2 = case["n2"]  # each unordered distance within a set and each between the sets once
    return {"bytes": 16.0 * (n + n2) + 24.0 * (n + n2), "flops": 5.0 * (n * n2 + 0.5 * n * n + 0.5 * n2 * n2)}


# ---------------------------------------------------------------------------
# the same results by plain torch in 64 bits
# ---------------------------------------------------------------------------
def _field(y, mu=MU):
    """Time derivative of (N, 6) states or (N, 42) STM + state rows."""
    s = y[:, -6:]
    x, v = s[:, :3], s[:, 3:]
    d1 = x + torch.tensor([mu, 0.0, 0.0], dtype=y.dtype, device=y.device)
    d2 = x - torch.tensor([1.0 - mu, 0.0, 0.0], dtype=y.dtype, device=y.device)
    q1, q2 = (d1 * d1).sum(1, keepdim=True), (d2 * d2).sum(1, keepdim=True)
    g1, g2 = (1.0 - mu) * q1 ** -1.5, mu * q2 ** -1.5
    plane = torch.tensor([1.0, 1.0, 0.0], dtype=y.dtype, device=y.device)
    cor = torch.stack((2.0 * v[:, 1], -2.0 * v[:, 0], torch.zeros_like(v[:, 0])), 1)
    a = x * plane + cor - g1 * d1 - g2 * d2
    if y.shape[1] == 6:
        return torch.cat((v, a), 1)
    eye = torch.eye(3, dtype=y.dtype, device=y.device)
    U = torch.diag(plane) - (g1 + g2)[:, :, None] * eye
    U = U + (3.0 * g1 / q1)[:, :, None] * d1[:, :, None] * d1[:, None, :]
    U = U + (3.0 * g2 / q2)[:, :, None] * d2[:, :, None] * d2[:, None, :]
    P = y[:, :36].reshape(-1, 6, 6)
    lo = (U[:, :, :, None] * P[:, None, :3, :]).sum(2)
    lo = lo + 2.0 * torch.stack((P[:, 4], -P[:, 3], torch.zeros_like(P[:, 3])), 1)
    return torch.cat((torch.cat((P[:, 3:], lo), 1).reshape(-1, 36), v, a), 1)


def _signed(fwd, dim):
    """The field of a backward run: the state's six derivatives negated (all
    of them for the 6-dim system; the package negates all 42 by default)."""
    return (lambda y: -_field(y)) if fwd < 0 else _field


def _extrapolate(f, y, H, columns=8):
    """One Gragg-Bulirsch-Stoer step of size H (scalar or (N, 1))."""
    table, counts = [], [2 * (k + 1) for k in range(columns)]
    for k, m in enumerate(counts):
        h = H / m
        a, b = y, y + h * f(y)
        for _ in range(m - 1):
            a, b = b, a + 2.0 * h * f(b)
        row = [0.5 * (a + b + h * f(b))]
        for j in range(1, k + 1):
            row.append(row[-1] + (row[-1] - table[j - 1]) / ((m / counts[k - j]) ** 2 - 1.0))
        table = row
    return table[-1]


def _solve(f, y, H, steps):
    out = [y]
    for _ in range(steps):
        out.append(_extrapolate(f, out[-1], H))
    return out


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "orbit":
        sub = 1 if case["m"] >= 250 else 4
        ys = _solve(_field, torch.as_tensor(_orbit_states(n, seed)), case["tf"] / (case["m"] - 1) / sub,
                    (case["m"] - 1) * sub)
        ys = torch.stack(ys[::sub])
        return {"y_end": ys[-1], "t_end": torch.full((n,), case["tf"], dtype=torch.float64), "n_accept": None,
                "n_reject": None, "status": None, "samples": ys}
    if kind == "fixed":
        if case["order"] == 4:
            y = workloads.stm_fixed_batch(n, seed=seed)
            y = _dev(y if case["dim"] == 42 else y[:, 36:])
            f, rows = _signed(case["fwd"], case["dim"]), [y]
            t = np.linspace(0.0, case["steps"] * 1e-3, case["steps"] + 1)
            for k in range(case["steps"]):
                h = float(t[k + 1] - t[k])
                k1 = f(y)
                k2 = f(y + 0.5 * h * k1)
                k3 = f(y + 0.5 * h * k2)
                k4 = f(y + h * k3)
                y = y + h / 6.0 * k1 + h / 3.0 * k2 + h / 3.0 * k3 + h / 6.0 * k4
                if (k + 1) % case["every"] == 0:
                    rows.append(y)
            return {"rows": torch.stack(rows), "status": None}
        return None  # some states pass close to a primary: the step size, not the solution, decides their digits
    if kind == "stability":
        y, T = _stability_inputs(n, seed)
        end = _solve(_field, _dev(y), _dev(T)[:, None] / 100.0, 100)[-1]
        return {"y_end": end, "t_end": _dev(T), "n_accept": None, "n_reject": None, "status": None,
                "samples": end[None]}
    if kind == "filters":
        s = prepare(case, seed)["samples"]
        x, v = s[..., :3], s[..., 3:]
        d1 = x + torch.tensor([MU, 0.0, 0.0], dtype=torch.float64, device=DEV)
        d2 = x - torch.tensor([1.0 - MU, 0.0, 0.0], dtype=torch.float64, device=DEV)
        r1, r2 = d1.square().sum(-1).sqrt(), d2.square().sum(-1).sqrt()
        C = x[..., 0] ** 2 + x[..., 1] ** 2 + 2.0 * ((1.0 - MU) / r1 + MU / r2) - v.square().sum(-1)
        return r1.amin(0), r2.amin(0), ((C - C[0]).abs() / C[0].abs()).amax(0)
    if kind == "pairs":
        pu, ps = (_dev(a) for a in _clouds(n, case["n2"], seed))

        def best(q, r):
            out = []
            for k in range(0, q.shape[0], 4096):
                dx, dy = q[k:k + 4096, :1] - r[None, :, 0], q[k:k + 4096, 1:] - r[None, :, 1]
                d2 = (dx * dx + dy * dy).amin(1)
                out.append(torch.where(d2 <= 1e-4 * 1e-4, d2, torch.zeros_like(d2)))
            return torch.cat(out)

        return {"us": (None, None, best(pu, ps)), "su": (None, None, best(ps, pu)), "u": None, "s": None}
    # adaptive runs to an event, corrections and detections: the step sequence
    # and the iteration define the result, which has no closed form
    return None

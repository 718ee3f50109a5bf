"""The work that users of this package have it do, as cases that can be timed
and compared: single steady solves, batches of steady solves, one large
steady system, time marching, harmonic balance, the strip-corrected solver,
and the two wake operators that a host's own time loop calls.

``listed()`` names the cases, ``draw(rng)`` gives another case of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call,
``run(state)`` is one pass through the public entry points, ``work(case)``
counts what the path cannot do without, and ``exact(case, seed)`` evaluates
the same quantities in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

from tinyvlm_gb300 import mesh as M
from tinyvlm_gb300.backend import Backend
from tinyvlm_gb300.batch import BatchSolver, pack_alphas, pack_verts
from tinyvlm_gb300.device import DeviceArray, PinnedArray
from tinyvlm_gb300.hbvlm import HBVLM2
from tinyvlm_gb300.kinematics import Assembly, KinematicsTree, rotation_matrix, sin, translation_matrix
from tinyvlm_gb300.uvlm import UVLM
from tinyvlm_gb300.vlm import NLVLM, VLM, Database, FlowData, WingProfile

TWO_PI_F = float(np.float32(2.0) * np.float32(3.141593))  # the solver's interface has a float pi
FOUR_PI = float(np.float32(4.0) * np.float32(3.141593))
EPS_F = 1.19209e-07
REF = (0.25, 0.0, 0.0)


def listed():
    return [
        # One VLM::run per call, as the reference's drivers call it: the 16 x 16 elliptic wing, float.
        # The smallest call: its latency is launches and short dependent chains.
        {"name": "vlm_f32_16x16", "kind": "vlm", "precision": 32, "nc": 16, "ns": 16},
        # The plain per-solve double path, the one users check the others against.
        {"name": "vlm_f64_20x45", "kind": "vlm", "precision": 64, "nc": 20, "ns": 45},
        # The headline: 512 uneven trapezoids, 8 angles each, one AIC per wing (a design-space sweep).
        {"name": "batch_shared_512x8", "kind": "batch", "mode": "shared", "count": 512, "alphas": 8},
        # The reference's alpha-dependent formulation, one AIC per wing and angle.
        {"name": "batch_exact_64x4", "kind": "batch", "mode": "exact", "count": 64, "alphas": 4},
        # One large wing, 64 angles on one AIC, circulations converged to the FP64 system's.
        {"name": "large_128x128x64", "kind": "large", "nc": 128, "ns": 128, "alphas": 64},
        # Pitch-plunge time marching, 1600 panels, 500 steps (the wake grows to 40,000 rings), float.
        {"name": "uvlm_f32_20x80x500", "kind": "uvlm", "precision": 32, "nc": 20, "ns": 80, "steps": 500},
        # The same in double on a coarser wing.
        {"name": "uvlm_f64_12x48x160", "kind": "uvlm", "precision": 64, "nc": 12, "ns": 48, "steps": 160},
        # One harmonic-balance solve of the pitch-heave section, as the continuation scripts call it.
        {"name": "hbvlm_45x1_h5", "kind": "hbvlm", "nc": 45, "harmonics": 5, "sets": 1},
        # The perturbed points of that section's finite-difference Jacobian, as one batch.
        {"name": "hbvlm_45x1_h5_x44", "kind": "hbvlm", "nc": 45, "harmonics": 5, "sets": 44},
        # The wake's influence on the right-hand side, called by a host's own time loop: 1600 points, 40,000 rings.
        {"name": "wake_rhs_f32_20x80x500", "kind": "wake_rhs", "precision": 32, "nc": 20, "ns": 80, "rows": 500},
        # One free-wake roll-up step of a wake of 150 rows.
        {"name": "rollup_f32_20x80x150", "kind": "rollup", "precision": 32, "nc": 20, "ns": 80, "rows": 150},
        # The strip-corrected (nonlinear) solver against a lift polar, 5 x 200 panels.
        {"name": "nlvlm_f32_5x200", "kind": "nlvlm", "nc": 5, "ns": 200},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["vlm", "batch", "large", "uvlm", "hbvlm", "wake_rhs", "rollup", "nlvlm"])
    if kind == "vlm":
        return {"kind": kind, "precision": rng.choice([32, 64]), "nc": _log(rng, 4, 32), "ns": _log(rng, 4, 64)}
    if kind == "batch":
        mode = rng.choice(["shared", "exact"])
        return {"kind": kind, "mode": mode, "count": _log(rng, 2, 512 if mode == "shared" else 96),
                "alphas": rng.randint(1, 8 if mode == "shared" else 4)}
    if kind == "large":
        return {"kind": kind, "nc": _log(rng, 40, 128), "ns": _log(rng, 40, 128), "alphas": _log(rng, 4, 64)}
    if kind == "uvlm":
        if rng.choice([32, 64]) == 32:
            return {"kind": kind, "precision": 32, "nc": _log(rng, 4, 20), "ns": _log(rng, 8, 80),
                    "steps": _log(rng, 40, 500)}
        return {"kind": kind, "precision": 64, "nc": _log(rng, 4, 12), "ns": _log(rng, 8, 48),
                "steps": _log(rng, 40, 160)}
    if kind == "hbvlm":
        return {"kind": kind, "nc": rng.randint(15, 45), "harmonics": rng.randint(1, 5), "sets": _log(rng, 1, 44)}
    if kind == "wake_rhs":
        p = rng.choice([32, 64])
        return {"kind": kind, "precision": p, "nc": _log(rng, 4, 20), "ns": _log(rng, 8, 80),
                "rows": _log(rng, 8, 500 if p == 32 else 200)}
    if kind == "rollup":
        p = rng.choice([32, 64])
        return {"kind": kind, "precision": p, "nc": _log(rng, 4, 20), "ns": _log(rng, 8, 80 if p == 32 else 40),
                "rows": _log(rng, 8, 150 if p == 32 else 60)}
    return {"kind": kind, "nc": _log(rng, 2, 8), "ns": _log(rng, 20, 200)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(case, seed):
    return np.random.Generator(np.random.PCG64([int(seed), 20261203]))


def _wing(rng, nc, ns):
    """A trapezoidal half wing over the ranges of the batched workload, quarter-chord shifted, float."""
    v = M.trapezoid(nc, ns, rng.uniform(4.0, 12.0), rng.uniform(0.3, 1.0), rng.uniform(0.0, 35.0)).astype(np.float32)
    M.quarter_chord(v)
    return v


def _steady_inputs(case, seed):
    rng = _rng(case, seed)
    if case["kind"] == "vlm":  # the elliptic planform, its root chord drawn; a small tip chord is not kept
        v = M.elliptic(case["nc"], case["ns"], 5.0, rng.uniform(0.8, 1.2)).astype(np.float32)
        if case["ns"] > 24 or case["precision"] == 64:  # finely spaced elliptic tips are slivers: a trapezoid there
            v = _wing(rng, case["nc"], case["ns"])
        else:
            M.quarter_chord(v)
        return v, math.radians(rng.uniform(1.0, 8.0))
    if case["kind"] == "nlvlm":
        v = M.rectangular(case["nc"], case["ns"], 1.0, rng.uniform(8.0, 20.0)).astype(np.float32)
        M.quarter_chord(v)
        alphas = np.linspace(0.0, math.radians(20.0), 100).astype(np.float32)
        cl0, a0, a1 = rng.uniform(0.7, 1.2), 0.28, rng.uniform(0.02, 0.04)
        cl = [2 * math.pi * a + 0.5 * (cl0 - 2 * math.pi * a) * (1.0 + math.erf((a - a0) / a1)) for a in alphas.tolist()]
        return v, math.radians(rng.uniform(4.0, 14.0)), alphas, np.array(cl, np.float32)
    if case["kind"] == "large":
        return [M.Case(_wing(rng, case["nc"], case["ns"]), np.radians(rng.uniform(-10.0, 10.0, case["alphas"])), {})]
    sizes = [(c.nc, c.ns) for c in _sizes(case["count"])]
    return [M.Case(_wing(rng, nc, ns), np.radians(rng.uniform(-8.0, 8.0, case["alphas"])), {}) for nc, ns in sizes]


_SIZES = {}


def _sizes(count):
    """The panel counts of the batched workload (its seed's); the wings themselves come from the case's seed."""
    if count not in _SIZES:
        _SIZES[count] = M.batch_cases(count, n_alpha=1)
    return _SIZES[count]


def _motion(seed):
    rng = np.random.Generator(np.random.PCG64([int(seed), 7]))
    return dict(k=rng.uniform(0.3, 0.7), h=rng.uniform(0.05, 0.15), th=math.radians(rng.uniform(1.0, 4.0)))


def _uvlm_inputs(case, seed):
    v = M.rectangular(case["nc"], case["ns"], 1.0, 4.0).astype(np.float32)
    M.quarter_chord(v)
    return v, _motion(seed), 1.0 / case["nc"]


def _hb_inputs(case, seed):
    rng = _rng(case, seed)
    v = M.rectangular(case["nc"], 1, 1.0, 40000.0)
    sets = []
    base = np.zeros((2, 2 * case["harmonics"] + 1))
    base[0, 1:3] = rng.uniform(-0.02, 0.02, 2)
    base[1, 0] = rng.uniform(-0.02, 0.02)
    base[1, 1:3] = rng.uniform(-0.04, 0.04, 2)
    omega = float(rng.uniform(0.2, 0.6))
    for s in range(case["sets"]):  # the point itself, then points that differ in one coefficient
        dyn = base.copy()
        if s:
            dyn.flat[(s - 1) % dyn.size] += (1.0 if s <= dyn.size else -1.0) * 1e-4
        sets.append(dyn)
    return v, omega, sets


def _wake_inputs(case, seed):
    """A wing mid-run in a host's time loop: its wake, shed by a heaving wing and already disturbed, with the
    circulations shed along it."""
    rng = _rng(case, seed)
    dt_ = np.float32 if case["precision"] == 32 else np.float64
    nc, ns, rows = case["nc"], case["ns"], case["rows"]
    wing = M.rectangular(nc, ns, 1.0, 4.0)
    M.quarter_chord(wing)
    nwv = rows + 1
    wake = np.zeros((4, nwv, ns + 1))
    wake[3] = 1.0
    age = np.arange(rows + 1, dtype=np.float64)  # row 0 is the newest, at the wing's trailing edge
    k, h, th = rng.uniform(0.3, 0.7), rng.uniform(0.05, 0.15), 0.05
    step = 1.0 / nc
    wake[0] = wing[0, -1][None, :] + (age * step)[:, None]
    wake[1] = wing[1, -1][None, :]
    wake[2] = (h * np.sin(k * age * step))[:, None]
    wake[:3, 1:] += rng.normal(0.0, 0.1 * step, (3, rows, ns + 1))
    y = (np.arange(ns) + 0.5) / ns
    load = np.sqrt(1.0 - y * y)[None, :]
    gwake = th * (1.0 + 0.5 * np.cos(k * age[:-1] * step))[:, None] * load
    gwing = th * ((np.arange(nc) + 1.0) / nc)[:, None] * load * rng.uniform(0.9, 1.1)
    return wing.astype(dt_), wake.astype(dt_), gwing.astype(dt_), gwake.astype(dt_)


def _dev(x):
    return DeviceArray.from_numpy(np.ascontiguousarray(x))


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _assembly(m):
    tree = KinematicsTree()
    fs = tree.add(lambda t: translation_matrix([-t, 0.0, 0.0]))
    heave = tree.add(lambda t: translation_matrix([0.0, 0.0, m["h"] * sin(m["k"] * t)])).after(fs)
    pitch = tree.add(lambda t: rotation_matrix([0.25, 0.0, 0.0], [0.0, 1.0, 0.0],
                                               m["th"] * sin(m["k"] * t + math.pi / 2))).after(heave)
    asm = Assembly(fs)
    asm.add("wing", pitch)
    return asm


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "vlm":
        v, alpha = _steady_inputs(case, seed)
        s.update(sim=VLM("gb300", [v], precision=case["precision"]), flow=FlowData(alpha))
    elif kind == "nlvlm":
        v, alpha, a, cl = _steady_inputs(case, seed)
        db = Database()
        db.profiles.append(WingProfile(a, cl))
        s.update(sim=NLVLM("gb300", [v]), flow=FlowData(alpha), db=db)
    elif kind in ("batch", "large"):
        cases = _steady_inputs(case, seed)
        bs = BatchSolver(cases, mode=case.get("mode", "shared"), refine=1, fp64_residual=kind == "large")
        verts = pack_verts(cases)
        pv = PinnedArray(verts.shape, np.float32)
        pv[:] = verts
        s.update(bs=bs, verts=pv, alphas=pack_alphas(cases), co=PinnedArray((bs.nsolve, 5), np.float64),
                 g=PinnedArray((bs.gamma_floats,), np.float32))
    elif kind == "uvlm":
        v, m, dt = _uvlm_inputs(case, seed)
        s.update(sim=UVLM("gb300", [v], precision=case["precision"]), asm=_assembly(m), dt=dt)
    elif kind == "hbvlm":
        v, omega, sets = _hb_inputs(case, seed)
        hb = HBVLM2("gb300", v)
        hb.init(case["harmonics"], 1.0)
        s.update(hb=hb, omega=omega, sets=sets)
    else:
        wing, wake, gwing, gwake = _wake_inputs(case, seed)
        be = Backend(wing.dtype)
        s.update(be=be, wing=_dev(wing), wake=_dev(wake), gwing=_dev(gwing), gwake=_dev(gwake))
        if kind == "wake_rhs":
            np_ = (3, case["nc"], case["ns"])
            s.update(colloc=DeviceArray(np_, wing.dtype), normals=DeviceArray(np_, wing.dtype),
                     areas=DeviceArray(np_[1:], wing.dtype),
                     rhs=torch.zeros(case["nc"] * case["ns"], device="cuda",
                                     dtype=torch.float32 if wing.dtype == np.float32 else torch.float64))
            be.mesh_metrics(0.0, [s["wing"]], [s["colloc"]], [s["normals"]], [s["areas"]])
        else:
            s.update(wake0=_dev(wake), out=torch.zeros((4,) + wake.shape[1:], device="cuda",
                                                       dtype=torch.float32 if wing.dtype == np.float32
                                                       else torch.float64))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "vlm":
        r, g = s["sim"].run(s["flow"], ref_pt=REF, return_gamma=True)
        co = np.array([r.cl, r.cd, *r.cm])
        # a precision=32 handle computes in float and reports its floats in double containers
        return (co, g) if case["precision"] == 64 else (co.astype(np.float32), g.astype(np.float32))
    if kind == "nlvlm":
        r = s["sim"].run(s["flow"], s["db"])
        return np.float32(r.cl), s["sim"].strip_alpha[0]
    if kind in ("batch", "large"):
        bs = s["bs"]
        bs.set_inputs(s["verts"], s["alphas"], ref_pt=REF)
        bs.run(want_gamma=True)
        bs.results_into(s["co"], s["g"])
        # coefficients summed (in double) over float circulations: kept as floats, like the circulations
        return np.asarray(s["co"]).astype(np.float32), np.asarray(s["g"])
    if kind == "uvlm":
        r = s["sim"].run(s["asm"], t_steps=case["steps"], dt=s["dt"], return_gamma=True)
        out = (r["cl"], r["cm"], r["gamma"])
        return out if case["precision"] == 64 else tuple(x.astype(np.float32) for x in out)
    if kind == "hbvlm":
        hb = s["hb"]
        hb.gamma_coeffs[:] = 0.0  # a solve from rest
        forces = [np.zeros((2, 2 * case["harmonics"] + 1)) for _ in s["sets"]]
        if len(forces) == 1:
            hb.run(s["omega"], s["sets"][0], forces[0])
        else:
            hb.run_batch([s["omega"]] * len(forces), s["sets"], forces)
        return np.stack(forces), np.ascontiguousarray(hb.gamma_coeffs)
    be = s["be"]
    if kind == "wake_rhs":
        s["rhs"].zero_()
        be.rhs_assemble_wake_influence(s["rhs"], [s["gwake"]], [s["colloc"]], [s["normals"]], [s["wake"]], [True],
                                       case["rows"])
        return s["rhs"]
    s["wake"].copy_from(s["wake0"])
    be.wake_rollup([s["wake"]], [s["wing"]], [s["gwing"]], [s["gwake"]], [True], 0.1 / case["nc"], case["rows"])
    be.memory.copy(0, s["out"].data_ptr(), 1, 0, s["wake"].data_ptr(), 1, 1, s["wake"].nbytes)
    return s["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# A lattice of rings costs each evaluation point, per ring, two segments (a ring's other two belong to its
# neighbours) and one vertex distance, each for the point and for its image in y = 0:
# 2 x (2 x 38 + 9) flops.
RING = 170.0


def work(case):
    kind = case["kind"]
    if kind in ("vlm", "nlvlm"):
        n = case["nc"] * case["ns"]
        size = 8 if case.get("precision") == 64 else 4
        return {"flops": RING * n * (n + case["ns"]) + 2 / 3 * n ** 3 + 2 * n * n,
                "bytes": 4 * 4 * (case["nc"] + 1) * (case["ns"] + 1) + size * (n + 5)}
    if kind in ("batch", "large"):
        sizes = [(case["nc"], case["ns"])] if kind == "large" else [(c.nc, c.ns) for c in _sizes(case["count"])]
        na = case["alphas"]
        per = na if case.get("mode") == "exact" else 1
        fl = by = 0.0
        for nc, ns in sizes:
            n = nc * ns
            fl += per * (RING * n * (n + ns) + 2 / 3 * n ** 3) + 3 * na * 2 * n * n
            by += 16 * (nc + 1) * (ns + 1) + na * (4 * n + 40 + 8)
        return {"flops": fl, "bytes": by}
    if kind == "uvlm":
        n, ns, t = case["nc"] * case["ns"], case["ns"], case["steps"]
        return {"flops": RING * n * n + 2 / 3 * n ** 3 + t * 2 * n * n + RING * n * ns * t * (t - 1) / 2,
                "bytes": 16 * (case["nc"] + 1) * (ns + 1) + t * (32 + 38 * 8) + n * case["precision"] / 8}
    if kind == "hbvlm":
        n, N = case["nc"], 2 * case["harmonics"] + 1
        rows = 3.5 * (2 * math.pi / 0.4) * case["nc"]
        return {"flops": case["sets"] * N * n * rows * (2 * RING + 2 * N), "bytes": 8 * case["sets"] * (2 + n) * N}
    n, ns, rows = case["nc"] * case["ns"], case["ns"], case["rows"]
    size = case["precision"] / 8
    if kind == "wake_rhs":
        return {"flops": RING * n * ns * rows, "bytes": size * (7 * n + 3 * (rows + 1) * (ns + 1) + rows * ns)}
    pts = rows * (ns + 1)
    return {"flops": RING * pts * (n + ns * rows), "bytes": size * (6 * (rows + 1) * (ns + 1) + rows * ns + 4 * n)}


# ---------------------------------------------------------------------------
# the same quantities in 64 bits, from the definitions
# ---------------------------------------------------------------------------
def _t(x):
    return torch.as_tensor(np.asarray(x, np.float64), device="cuda" if torch.cuda.is_available() else "cpu")


def _segments(P, A, B):
    """k and c = (B - A) x (P - A) with 4 pi v = k c, of the segments A -> B at the points P (broadcast against
    each other): Katz and Plotkin eq. 10.115 with nothing that cancels, and its cut-offs."""
    r0 = [B[..., i] - A[..., i] for i in range(3)]
    a = [P[..., i] - A[..., i] for i in range(3)]
    b = [P[..., i] - B[..., i] for i in range(3)]
    c = [r0[1] * a[2] - r0[2] * a[1], r0[2] * a[0] - r0[0] * a[2], r0[0] * a[1] - r0[1] * a[0]]
    an = (a[0] * a[0] + a[1] * a[1] + a[2] * a[2]).sqrt_()
    bn = (b[0] * b[0] + b[1] * b[1] + b[2] * b[2]).sqrt_()
    ab = a[0] * b[0] + a[1] * b[1] + a[2] * b[2]
    sq = c[0] * c[0] + c[1] * c[1] + c[2] * c[2]
    m = an * bn
    k = torch.where(ab >= 0, (an + bn) / (m * (m + ab)), (an + bn) * (m - ab) / (m * sq))
    return torch.where((sq < 1e-10) | (an < 1e-10) | (bn < 1e-10), torch.zeros_like(k), k), c


_FLIP = torch.tensor([1.0, -1.0, 1.0], dtype=torch.float64)


def _velocity(P, V, G, most=1 << 24):
    """4 pi times the velocity at the points P (n, 3) of the lattice V (rows + 1, ns + 1, 3) with ring strengths
    G (rows, ns), and of its image in y = 0: each segment once, with the difference of its two rings' strengths."""
    z = torch.zeros_like(G[:1])
    gs = torch.cat([G, z]) - torch.cat([z, G])  # along the span, line j: the ring below it less the one above
    zc = torch.zeros_like(G[:, :1])
    gc = torch.cat([zc, G], 1) - torch.cat([G, zc], 1)  # along the chord, vertex k: right of ring k - 1, left of k
    out = torch.zeros_like(P)
    step = max(1, most // V[..., 0].numel())
    flip = _FLIP.to(P.device)
    for i in range(0, P.shape[0], step):
        for f in (None, flip):
            p = P[i:i + step] if f is None else P[i:i + step] * f
            vel = 0.0
            for A, B, g in ((V[:, :-1], V[:, 1:], gs), (V[:-1], V[1:], gc)):
                k, c = _segments(p[:, None, None, :], A, B)
                k *= g
                vel = vel + torch.stack([(k * x).sum((1, 2)) for x in c], 1)
            out[i:i + step] += vel if f is None else vel * f
    return out


def _aic(P, N, V, most=1 << 24):
    """4 pi times the normal velocity at P of every ring of V with its image, at unit strength: (n, rows, ns)."""
    R, S = V.shape[0] - 1, V.shape[1] - 1
    out = torch.empty((P.shape[0], R, S), dtype=torch.float64, device=P.device)
    step = max(1, most // V[..., 0].numel())
    flip = _FLIP.to(P.device)
    for i in range(0, P.shape[0], step):
        o = 0.0
        for f in (None, flip):
            p, n = (P[i:i + step], N[i:i + step]) if f is None else (P[i:i + step] * f, N[i:i + step] * f)
            val = []
            for A, B in ((V[:, :-1], V[:, 1:]), (V[:-1], V[1:])):
                k, c = _segments(p[:, None, None, :], A, B)
                val.append(k * sum(c[q] * n[:, None, None, q] for q in range(3)))
            o = o + val[0][:, :-1] - val[0][:, 1:] + val[1][:, :, 1:] - val[1][:, :, :-1]
        out[i:i + step] = o
    return out


def _lattice(v):
    return _t(np.moveaxis(np.asarray(v, np.float64)[:3], 0, -1))


def _metrics(V, alpha=0.0):
    """Collocation points, normals (rows, ns, 3) and areas of a lattice."""
    f = 0.5 if alpha < EPS_F else 0.5 * (alpha / (math.sin(alpha) + EPS_F))
    v0, v1, v2, v3 = V[:-1, :-1], V[:-1, 1:], V[1:, 1:], V[1:, :-1]
    n = torch.linalg.cross(v3 - v1, v2 - v0)
    n = n / n.norm(dim=-1, keepdim=True)
    area = 0.5 * (torch.linalg.cross(v3 - v0, v2 - v0).norm(dim=-1) + torch.linalg.cross(v2 - v0, v1 - v0).norm(dim=-1))
    return 0.5 * (v0 + v1) + f * 0.5 * (v2 + v3 - v0 - v1), n, area


def _delta(g):
    return torch.cat([g[:1], g[1:] - g[:-1]])


def _mac(V, area):
    c = (V[0] - V[-1]).norm(dim=-1)
    w = (V[0, 1:] - V[0, :-1]).norm(dim=-1)
    return (0.5 * (c[:-1] ** 2 + c[1:] ** 2) * w).sum() / area.sum()


def _cl_cm(V, F, area, fs, ref):
    lift = np.array([-fs[2], 0.0, fs[0]])
    lift = _t(lift / np.linalg.norm(lift))
    q = 0.5 * float(np.dot(fs, fs)) * area.sum()
    lever = 0.5 * (V[:-1, :-1] + V[:-1, 1:]) - _t(ref)
    return (F @ lift).sum() / q, torch.linalg.cross(lever, F).sum((0, 1)) / (q * _mac(V, area))


def _stream(alpha):
    return np.array([math.cos(alpha), 0.0, math.sin(alpha)])


def _wake_ring(V, alpha):
    return torch.stack([V[-1], V[-1] + 100.0 * _t(_stream(alpha))])


def _trefftz(W):
    """K with CDi = g K g / area: the trailing segments of the ring row W = (trailing edge, 100 chords behind),
    seen from the rings' centres."""
    near, far = W[0], W[1]
    c = 0.25 * (near[:-1] + near[1:] + far[1:] + far[:-1])
    n = torch.linalg.cross(far[:-1] - near[1:], far[1:] - near[:-1])
    n = n / n.norm(dim=-1, keepdim=True)
    K = 0.0
    flip = _FLIP.to(W.device)
    for f in (None, flip):
        p, q = (c, n) if f is None else (c * f, n * f)
        for A, B in ((near[1:], far[1:]), (far[:-1], near[:-1])):
            k, x = _segments(p[:, None, :], A, B)
            K = K + k * sum(x[i] * q[:, None, i] for i in range(3))
    return -K / FOUR_PI * (near[1:] - near[:-1]).norm(dim=-1)[:, None]


def _factored(V, alpha):
    """Collocation data and the factors of the steady system (the wake row hangs on the trailing-edge rings)."""
    col, nor, area = _metrics(V, alpha)
    P, N = col.reshape(-1, 3), nor.reshape(-1, 3)
    A = _aic(P, N, V)
    A[:, -1] += _aic(P, N, _wake_ring(V, alpha))[:, 0]
    n = P.shape[0]
    return nor, area, torch.linalg.lu_factor((A / FOUR_PI).reshape(n, n))


def _steady(V, factored, alphas, wake_alpha=None):
    nor, area, lu = factored
    nc, ns = area.shape
    fs = [_stream(a) for a in alphas]
    rhs = torch.stack([-(nor.reshape(-1, 3) @ _t(f)) for f in fs], 1)
    G = torch.linalg.lu_solve(lu[0], lu[1], rhs)
    co = []
    for q, f in enumerate(fs):
        g = G[:, q].reshape(nc, ns)
        F = _delta(g)[..., None] * torch.linalg.cross(_t(f).expand(nc, ns, 3), V[:-1, 1:] - V[:-1, :-1])
        cl, cm = _cl_cm(V, F, area, f, REF)
        te = g[-1]
        cd = te @ (_trefftz(_wake_ring(V, 0.0 if wake_alpha is None else wake_alpha)) @ te) / area.sum()
        co.append(torch.cat([cl[None], cd[None], cm]))
    return torch.stack(co), G.T


def _pose(m, t):
    """4 x 4 transform of the pitch-plunge motion and its rate at the times t."""
    t = np.atleast_1d(np.asarray(t, np.float64))
    th = m["th"] * np.sin(m["k"] * t + math.pi / 2)
    thd = m["th"] * m["k"] * np.cos(m["k"] * t + math.pi / 2)
    return _section(th, thd, 0.25, -t, -np.ones_like(t), m["h"] * np.sin(m["k"] * t), m["h"] * m["k"] * np.cos(m["k"] * t))


def _section(th, thd, px, x, xd, z, zd):
    """Rotation by th about the y axis through (px, 0, 0), then the translation (x, 0, z); and its rate."""
    T = np.zeros((th.size, 4, 4))
    D = np.zeros_like(T)
    c, s = np.cos(th), np.sin(th)
    T[:, 0, 0] = T[:, 2, 2] = c
    T[:, 0, 2], T[:, 2, 0] = s, -s
    T[:, 1, 1] = T[:, 3, 3] = 1.0
    T[:, 0, 3], T[:, 2, 3] = px - c * px + x, s * px + z
    D[:, 0, 0] = D[:, 2, 2] = -s * thd
    D[:, 0, 2], D[:, 2, 0] = c * thd, -c * thd
    D[:, 0, 3], D[:, 2, 3] = s * thd * px + xd, c * thd * px + zd
    return T, D


def _move(T, V):
    T = _t(T)
    return V @ T[:3, :3].T + T[:3, 3]


def _exact_uvlm(case, seed):
    v, m, dt = _uvlm_inputs(case, seed)
    steps = case["steps"]
    T, D = _pose(m, np.arange(steps + 1) * dt)
    V0 = _move(T[0], _lattice(v))
    V = V0
    col, nor, area = _metrics(V)
    col0 = col
    nc, ns = area.shape
    n = nc * ns
    lu = torch.linalg.lu_factor((_aic(col.reshape(-1, 3), nor.reshape(-1, 3), V) / FOUR_PI).reshape(n, n))
    lines, strengths = [], []  # oldest first
    prev = torch.zeros_like(area)
    cl, cm = np.zeros(steps), np.zeros((steps, 3))
    for i in range(steps - 1):
        lines.append(V[-1])
        vel = -(col0 @ _t(D[i][:3, :3]).T + _t(D[i][:3, 3]))
        rhs = -(vel * nor).sum(-1).reshape(-1)
        if i:
            # newest line first: the ring between the lines of steps i - 1 and i carries step i - 1's strength
            w = _velocity(col.reshape(-1, 3), torch.stack(lines[::-1]), torch.stack(strengths[::-1]))
            rhs = rhs - (w * nor.reshape(-1, 3)).sum(-1) / FOUR_PI
        g = torch.linalg.lu_solve(lu[0], lu[1], rhs[:, None])[:, 0].reshape(nc, ns)
        strengths.append(g[-1])
        if i:
            F = _delta(g)[..., None] * torch.linalg.cross(vel, V[:-1, 1:] - V[:-1, :-1])
            F = F + ((g - prev) / dt * area)[..., None] * nor
            c, x = _cl_cm(V, F, area, np.array([1.0, 0.0, 0.0]), (T[i] @ np.array([0.5, 0.0, 0.0, 1.0]))[:3])
            cl[i], cm[i] = float(c), x.cpu().numpy()
        prev = g
        V = _move(T[i + 1], V0)
        col, nor, _ = _metrics(V)
    return cl, cm, prev.reshape(-1)


def _exact_hbvlm(case, seed):
    v, omega, sets = _hb_inputs(case, seed)
    V0 = _lattice(v)
    H = case["harmonics"]
    U = 2 * H + 1
    col_h, nor_h, _ = _metrics(V0)
    nc, ns = nor_h.shape[:2]
    n = nc * ns
    P0 = col_h.reshape(-1, 3)
    lu = torch.linalg.lu_factor((_aic(P0, nor_h.reshape(-1, 3), V0) / FOUR_PI).reshape(n, n))
    chord = float((V0[-1, 0] - V0[-2, 0]).norm())
    period = TWO_PI_F / omega
    interval = period / U
    dt = interval / math.ceil(interval / chord)
    t_start = 3.0 * TWO_PI_F / omega
    max_t = int((t_start + period + dt) / dt)
    ts = [int(round((t_start + period * q / U) / dt)) for q in range(U)]
    fts = [int(round(period * q / U / dt)) for q in range(U)]
    s0, s2 = 1.0 / math.sqrt(U), math.sqrt(2.0 / U)
    tq = np.arange(U) / U * period
    dft, ddft = np.full((U, U), s0), np.zeros((U, U))
    for h in range(H):
        w = omega * (h + 1)
        dft[:, 2 * h + 1], dft[:, 2 * h + 2] = np.cos(w * tq) * s2, np.sin(w * tq) * s2
        ddft[:, 2 * h + 1], ddft[:, 2 * h + 2] = -w * np.sin(w * tq) * s2, w * np.cos(w * tq) * s2

    def pose(dyn, t):
        def series(r):
            val, rate = np.full_like(t, r[0]), np.zeros_like(t)
            for h in range(H):
                w = omega * (h + 1)
                val = val + np.cos(w * t) * r[2 * h + 1] + np.sin(w * t) * r[2 * h + 2]
                rate = rate - w * np.sin(w * t) * r[2 * h + 1] + w * np.cos(w * t) * r[2 * h + 2]
            return val, rate
        (h0, h1), (p0, p1) = series(dyn[0]), series(dyn[1])
        return _section(p0, p1, 0.5, -t, -np.ones_like(t), -h0, -h1)

    forces, X = [], None
    for dyn in sets:
        Tw, _ = pose(dyn, np.arange(max_t) * dt)
        Tw = _t(Tw)
        lines = torch.einsum("tij,kj->tki", Tw[:, :3, :3], V0[-1]) + Tw[:, None, :3, 3]  # by step: oldest first
        Ti, Di = pose(dyn, np.array(ts) * dt)
        c0, L = [], []
        for q in range(U):
            V = _move(Ti[q], V0)
            col, nor, _ = _metrics(V)
            N = nor.reshape(-1, 3)
            vel = -(col_h @ _t(Di[q][:3, :3]).T + _t(Di[q][:3, 3]))
            c0.append(-(vel.reshape(-1, 3) * N).sum(-1))
            it = ts[q]
            # ring row r (0: the newest of `it`) lies between the lines of steps it - 1 - r and it - r
            back = np.arange(it) + 1.0
            W = lines[:it + 1].flip(0)
            B = np.full((it, U), s0)
            for h in range(H):
                w = omega * (h + 1)
                ph = w * (ts[q] * dt - back * dt)
                B[:, 2 * h + 1], B[:, 2 * h + 2] = np.cos(ph) * s2, np.sin(ph) * s2
            ring = _aic(col.reshape(-1, 3), N, W)  # (n, it, ns)
            L.append(-torch.einsum("pri,rc->pic", ring, _t(B)) / FOUR_PI)
        D = _t(dft)
        c0 = torch.linalg.lu_solve(lu[0], lu[1], torch.stack(c0, 1) @ D)  # (n, U)
        L = torch.einsum("qpic,qd->pdic", torch.stack(L), D).reshape(n, U * ns * U)
        L = torch.linalg.lu_solve(lu[0], lu[1], L).reshape(n, U, ns, U)
        te = L[n - ns:].reshape(ns, U, ns, U).reshape(ns * U, ns * U)
        x = torch.linalg.solve(torch.eye(ns * U, dtype=torch.float64, device=te.device) - te, c0[n - ns:].reshape(-1))
        X = c0 + torch.einsum("pdic,ic->pd", L, x.reshape(ns, U))
        Tf, Df = pose(dyn, np.array(fts) * dt)
        f = np.zeros((2, U))
        for q in range(U):
            V = _move(Tf[q], V0)
            col, nor, area = _metrics(V)
            vel = -(col_h @ _t(Df[q][:3, :3]).T + _t(Df[q][:3, 3]))
            g, dg = (X @ _t(dft[q])).reshape(nc, ns), (X @ _t(ddft[q])).reshape(nc, ns)
            F = _delta(g)[..., None] * torch.linalg.cross(vel, V[:-1, 1:] - V[:-1, :-1]) + (dg * area)[..., None] * nor
            cl, cm = _cl_cm(V, F, area, np.array([1.0, 0.0, 0.0]), (Tf[q] @ np.array([0.5, 0.0, 0.0, 1.0]))[:3])
            f[0, q], f[1, q] = float(cl), float(cm[1])
        forces.append(f)
    return np.stack(forces), X


def _akima(x, y):
    m = np.diff(y) / np.diff(x)
    s = np.zeros_like(y)
    s[0], s[1], s[-2], s[-1] = m[0], 0.5 * (m[0] + m[1]), 0.5 * (m[-2] + m[-1]), m[-1]
    for i in range(2, len(x) - 2):
        a, b = abs(m[i + 1] - m[i]), abs(m[i - 1] - m[i - 2])
        s[i] = (a * m[i - 1] + b * m[i]) / (a + b) if a + b > 0 else 0.5 * (m[i] + m[i - 1])

    def at(q):
        i = np.clip(np.searchsorted(x, q, side="left") - 1, 0, len(x) - 2)
        d, u = x[i + 1] - x[i], q - x[i]
        c3 = (3 * m[i] - 2 * s[i] - s[i + 1]) / d
        c4 = (s[i] + s[i + 1] - 2 * m[i]) / (d * d)
        r = y[i] + s[i] * u + c3 * u * u + c4 * u ** 3
        return np.where(q <= x[0], y[0] - m[0] * (x[0] - q), np.where(q > x[-1], y[-1] + m[-1] * (q - x[-1]), r))
    return at


def _exact_nlvlm(case, seed):
    v, alpha, a, cl = _steady_inputs(case, seed)
    V = _lattice(v)
    nor, area, lu = _factored(V, alpha)
    nc, ns = area.shape
    at = _akima(a.astype(np.float64), cl.astype(np.float64))
    strip = np.full(ns, alpha)
    sarea = area.sum(0).cpu().numpy()
    bound = (V[:-1, 1:] - V[:-1, :-1])
    err, it = 1.0, 0
    while it < 100 and err > 1e-5:
        fs = np.stack([np.cos(strip), 0 * strip, np.sin(strip)], 1)
        vel = _t(fs)[None].expand(nc, ns, 3)
        g = torch.linalg.lu_solve(lu[0], lu[1], -(vel * nor).sum(-1).reshape(-1, 1)).reshape(nc, ns)
        F = (_delta(g)[..., None] * torch.linalg.cross(vel, bound)).sum(0).cpu().numpy()
        c = (-F[:, 0] * fs[:, 2] + F[:, 2] * fs[:, 0]) / (0.5 * sarea)
        corr = (at(c / TWO_PI_F - strip + alpha) - c) / TWO_PI_F
        strip = strip + corr
        err = np.abs(corr).sum() / (nc * ns)
        it += 1
    f = _stream(alpha)
    F = _delta(g)[..., None] * torch.linalg.cross(_t(f).expand(nc, ns, 3), bound)
    return float(_cl_cm(V, F, area, f, REF)[0]), strip


def exact(case, seed):
    kind = case["kind"]
    if kind == "vlm":
        v, alpha = _steady_inputs(case, seed)
        V = _lattice(v)
        co, g = _steady(V, _factored(V, alpha), [alpha], alpha)
        return co[0], g[0]
    if kind in ("batch", "large"):
        cos, gs = [], []
        for c in _steady_inputs(case, seed):
            V = _lattice(c.verts)
            if case.get("mode") == "exact":
                for a in c.alphas:
                    co, g = _steady(V, _factored(V, float(a)), [float(a)], float(a))
                    cos.append(co)
                    gs.append(g.reshape(-1))
            else:
                co, g = _steady(V, _factored(V, 0.0), [float(a) for a in c.alphas])
                cos.append(co)
                gs.append(g.reshape(-1))
        return torch.cat(cos), torch.cat(gs)
    if kind == "uvlm":
        return _exact_uvlm(case, seed)
    if kind == "hbvlm":
        return _exact_hbvlm(case, seed)
    if kind == "nlvlm":
        return _exact_nlvlm(case, seed)
    wing, wake, gwing, gwake = _wake_inputs(case, seed)
    V, W, GW, GK = _lattice(wing), _lattice(wake), _t(gwing), _t(gwake)
    if kind == "wake_rhs":
        # the points are the float (or double) ones that the solver's own geometry call makes of the float wing
        col, nor, _ = _metrics(V)
        P, N = col.reshape(-1, 3), nor.reshape(-1, 3)
        return -(_velocity(P, W, GK) * N).sum(-1) / FOUR_PI
    P = W[1:].reshape(-1, 3)
    vel = _velocity(P, V, GW) + _velocity(P, W, GK)
    out = _t(wake).clone()
    out[:3, 1:] += (0.1 / case["nc"] / FOUR_PI * vel).reshape(W[1:].shape).movedim(-1, 0)
    return out

"""The workloads that this library's speed is judged by.

Every case is a dict of plain values; ``listed`` gives the fixed ones,
``draw`` one more of the same ranges.  ``prepare`` makes what a program holds
before the call (positions, loads, a context, a solver or a simulation),
``run`` makes one pass through the public entry points, ``work`` counts what a
pass cannot do without, and ``exact`` gives the same results from plain torch
in 64 bits.

Kinds:

* ``segments``: M_ss, segment forces and torques to velocities, free space;
* ``wall``: M_ss above a no-slip wall;
* ``blobs``: M_bb, blob forces to velocities, in each of the three precisions;
* ``coupling``: M_bs and M_sb of one swimmer, the two directions between its
  segments and its blobs;
* ``barrier``: the short-range barrier forces of one swimmer;
* ``solve``: one mobility problem of a rigid body with its filaments
  (barrier, pair sums, GMRES for the blob forces and the body velocity);
* ``step``: one implicit time step of a swimmer.

Radii and viscosity are 1 unless a case says otherwise, segments are 2.2
apart along a filament, and filaments have 20 segments, as in the package's
workloads.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from generic_mobility_interface_class_gb300 import seeding, workloads
from generic_mobility_interface_class_gb300._lib import GMI_DF64, GMI_FP32C, GMI_FP64
from generic_mobility_interface_class_gb300.mobility import Context
from generic_mobility_interface_class_gb300.sim import Simulation
from generic_mobility_interface_class_gb300.solver import MobilitySolver

PRECISION = {"fp64": GMI_FP64, "fp32c": GMI_FP32C, "df64": GMI_DF64}
NSEG = 20
DL = 2.2
F64 = torch.float64
# typical GMRES iterations of one solve and residual evaluations and GMRES
# iterations of one step, for the operation counts of `work`
SOLVE_ITERATIONS, STEP_EVALUATIONS, STEP_ITERATIONS = 30, 6, 225


def listed():
    return [
        # the smallest call in use: the segments of the 962-particle swimmer
        dict(name="segments-320-fp64", kind="segments", precision="fp64", n=320, layout="swimmer"),
        # the segments of the 16,896-particle swimmer, in the default precision
        dict(name="segments-12800-fp64", kind="segments", precision="fp64", n=12800, layout="swimmer"),
        # a few filaments more than the warp-per-target range, an odd count
        dict(name="segments-2501-fp32c", kind="segments", precision="fp32c", n=2501, layout="swimmer"),
        # the benchmark's apply: a random suspension
        dict(name="segments-131072-fp32c", kind="segments", precision="fp32c", n=131072, layout="cloud"),
        # a carpet of 64 filaments on a wall
        dict(name="wall-1280-fp64", kind="wall", precision="fp64", n=1280),
        # the blob-blob operator of the 16,896-particle swimmer's GMRES solve
        dict(name="blobs-4096-fp64", kind="blobs", precision="fp64", n=4096, rblob=1.0),
        # the same operator in the precision of the refinement's residual, at the 10,242-blob body
        dict(name="blobs-10242-df64", kind="blobs", precision="df64", n=10242, rblob=1.0),
        # and in the precision of the refinement's inner solves
        dict(name="blobs-10242-fp32c", kind="blobs", precision="fp32c", n=10242, rblob=1.0),
        # segments <-> blobs of the 16,896-particle swimmer
        dict(name="coupling-12800-4096-fp64", kind="coupling", precision="fp64", n=12800, nblob=4096, rblob=1.0),
        # barrier forces of the 16,896-particle swimmer
        dict(name="barrier-16896", kind="barrier", precision="fp64", n=12800, nblob=4096),
        # one mobility problem of the 962-particle swimmer, as the reference's main loop asks for it
        dict(name="solve-962-fp64", kind="solve", precision="fp64", nfil=16, nblob=642, radius=10.0),
        # one implicit time step of the 16,896-particle swimmer
        dict(name="step-16896-fp32c", kind="step", precision="fp32c", nfil=640, nblob=4096, radius=40.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["segments", "segments", "segments", "wall", "blobs", "blobs", "blobs", "coupling", "barrier",
                       "solve", "step"])
    if kind == "segments":
        precision = rng.choice(["fp64", "fp32c"])
        n = _log_int(rng, 40, 13000 if precision == "fp64" else 131072)
        return dict(kind=kind, precision=precision, n=n, layout=rng.choice(["swimmer", "cloud"]))
    if kind == "wall":
        return dict(kind=kind, precision=rng.choice(["fp64", "fp32c"]), n=_log_int(rng, 60, 5000))
    if kind == "blobs":
        return dict(kind=kind, precision=rng.choice(["fp64", "fp32c", "df64"]), n=_log_int(rng, 42, 10242),
                    rblob=rng.choice([1.0, 1.0, 0.75, 1.3]))
    if kind == "coupling":
        return dict(kind=kind, precision=rng.choice(["fp64", "fp32c"]), n=_log_int(rng, 40, 12800),
                    nblob=_log_int(rng, 42, 4096), rblob=rng.choice([1.0, 1.0, 0.75, 1.3]))
    if kind == "barrier":
        return dict(kind=kind, precision="fp64", n=_log_int(rng, 100, 40000), nblob=_log_int(rng, 42, 10242))
    radius = rng.uniform(10.0, 20.0) if kind == "solve" else rng.uniform(10.0, 40.0)
    nblob = int(round(642 + (4096 - 642) * (radius - 10.0) / 30.0))  # as the package's uneven swimmers
    nfil = min(_log_int(rng, 8, 512), workloads.max_filaments(radius))
    return dict(kind=kind, precision="fp64" if kind == "solve" else "fp32c", nfil=nfil, nblob=nblob, radius=radius)


# ---- inputs -------------------------------------------------------------------
def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    return q * np.sign(np.diag(r))


def _body_radius(nblob):
    """The radius at which nblob blobs cover a sphere as 4096 cover one of 40."""
    return 40.0 * math.sqrt(nblob / 4096.0)


def _filaments(rng, n, radius, bend=3.0):
    """n segments (n, 3) of 20-segment filaments standing on a sphere, each bent sideways by up to `bend` at its tip."""
    nfil = -(-n // NSEG)
    dirs = seeding.fibonacci_sphere(nfil) @ _rotation(rng).T
    x = seeding.radial_filaments(dirs, radius + 1.05 * (0.5 * DL + 1.0), NSEG, DL).reshape(nfil, NSEG, 3)
    side = np.cross(dirs, rng.normal(size=(nfil, 3)))
    side *= rng.uniform(0.0, bend, size=(nfil, 1)) / np.maximum(np.linalg.norm(side, axis=1, keepdims=True), 1e-9)
    s = np.linspace(0.0, 1.0, NSEG) ** 2
    return (x + s[None, :, None] * side[:, None, :]).reshape(-1, 3)[:n].copy()


def _cloud(rng, n):
    """n particles at volume fraction 0.05, no two closer than 2.2: a shuffled cubic lattice with jitter."""
    pitch = (4.0 / 3.0 * math.pi / 0.05) ** (1.0 / 3.0)
    side = math.ceil(round(n ** (1.0 / 3.0), 9))
    cell = rng.permutation(side ** 3)[:n]
    x = np.stack([cell % side, cell // side % side, cell // (side * side)], axis=1).astype(np.float64) * pitch
    jitter = 0.5 * (pitch - 2.2)
    return x + rng.uniform(-jitter, jitter, size=(n, 3))


def _carpet(rng, n):
    """n segments of 20-segment filaments standing on the wall z = 0 on a grid 6 apart, bent sideways."""
    nfil = -(-n // NSEG)
    side = math.ceil(math.sqrt(nfil))
    base = 6.0 * np.stack([np.arange(nfil) % side, np.arange(nfil) // side], axis=1)
    angle = rng.uniform(0.0, 2.0 * math.pi, size=nfil)
    tip = rng.uniform(0.0, 3.0, size=nfil)
    s = np.linspace(0.0, 1.0, NSEG) ** 2
    x = np.empty((nfil, NSEG, 3))
    x[:, :, 0] = base[:, 0:1] + s[None, :] * (tip * np.cos(angle))[:, None]
    x[:, :, 1] = base[:, 1:2] + s[None, :] * (tip * np.sin(angle))[:, None]
    x[:, :, 2] = 1.5 + DL * np.arange(NSEG)[None, :]
    return x.reshape(-1, 3)[:n].copy()


def _inputs(case, seed):
    """The case's arrays on the host: positions and loads."""
    rng = np.random.default_rng(seed)
    kind, n = case["kind"], case.get("n")
    if kind == "segments":
        x = _cloud(rng, n) if case["layout"] == "cloud" else _filaments(rng, n, _body_radius(0.32 * n))
        return dict(xs=x, fs=rng.normal(size=(n, 6)))
    if kind == "wall":
        return dict(xs=_carpet(rng, n), fs=rng.normal(size=(n, 6)))
    if kind == "blobs":
        rot = _rotation(rng).T
        return dict(xb=_body_radius(n) * seeding.fibonacci_sphere(n) @ rot, fb=rng.normal(size=(n, 3)))
    if kind in ("coupling", "barrier"):
        radius = _body_radius(case["nblob"])
        xs = _filaments(rng, n, radius, bend=15.0 if kind == "barrier" else 3.0)
        rot = _rotation(rng).T
        return dict(xs=xs, fs=rng.normal(size=(n, 6)), xb=radius * seeding.fibonacci_sphere(case["nblob"]) @ rot,
                    fb=rng.normal(size=(case["nblob"], 3)))
    # solve: the body's blobs, the filaments, an external force and torque, and the loads of two successive calls
    radius = case["radius"]
    return dict(refs=radius * seeding.fibonacci_sphere(case["nblob"]),
                xs=_filaments(rng, case["nfil"] * NSEG, radius), body_f=10.0 * rng.normal(size=(1, 6)),
                loads=rng.normal(size=(2, case["nfil"] * NSEG, 6)))


def _seg_scale(case):
    return 2.0 * workloads.instability_parameters(NSEG)["end_force_magnitude"]


def prepare(case, seed):
    kind = case["kind"]
    precision = PRECISION[case["precision"]]
    if kind == "step":
        base = case["radius"] + 1.05 * (0.5 * DL + 1.0)
        fils = workloads.random_surface_points(case["nfil"], 2.0 * DL / base, seed)
        kw = workloads.free_swimmer(seeding.fibonacci_sphere(case["nblob"]), fils, radius=case["radius"], nseg=NSEG,
                                    seed=seed)
        sim = Simulation(**kw, precision=precision)
        sim.prepare()
        for _ in range(3):  # past the first steps from a straight start, which cost the most and stand for the least
            sim.step()
        return dict(kind=kind, sim=sim)
    host = _inputs(case, seed)
    if kind == "solve":
        phys = workloads.instability_parameters(NSEG)
        solver = MobilitySolver(nswim=1, nfil=case["nfil"], nseg=NSEG, nblob=case["nblob"],
                                repulsive_force_factor=phys["repulsive_force_factor"],
                                end_force_magnitude=phys["end_force_magnitude"], linear_tol=1e-8, precision=precision)
        solver.set_blob_references(host["refs"])
        solver.x_segs_host[:] = host["xs"]
        solver.f_segs_host[:] = 0.0
        body_x, body_q = np.zeros((1, 3)), np.array([[1.0, 0.0, 0.0, 0.0]])
        solver.make_body_reference_matrices(body_x, body_q)
        return dict(kind=kind, solver=solver, body_x=body_x, body_q=body_q, xs=host["xs"], loads=host["loads"],
                    body_f=host["body_f"], calls=0)
    state = {k: torch.as_tensor(np.ascontiguousarray(v), device="cuda") for k, v in host.items()}
    return dict(state, kind=kind, ctx=Context(0, precision), rblob=case.get("rblob", 1.0), scale=_seg_scale(case))


def run(state):
    kind = state["kind"]
    if kind == "step":
        sim = state["sim"]
        sim.step()
        return {k: sim.state(k) for k in ("seg_x", "seg_q", "seg_v", "body_x", "body_q", "body_v")}
    if kind == "solve":
        # each call of a time step has new forces; the last solution is the warm start
        solver = state["solver"]
        solver.x_segs_host[:] = state["xs"]
        solver.f_segs_host[:] = state["loads"][state["calls"] % 2]
        state["calls"] += 1
        _, body_f = solver.compute_velocities(state["body_x"], state["body_q"], state["body_f"])
        return dict(v_segs=solver.v_segs_host, f_blobs=solver.f_blobs_host, v_bodies=solver.v_bodies(), body_f=body_f)
    ctx = state["ctx"]
    if kind == "segments":
        return ctx.mss(state["xs"], state["fs"])
    if kind == "wall":
        return ctx.mss_wall(state["xs"], state["fs"])
    if kind == "blobs":
        return ctx.mbb(state["xb"], state["fb"], a=state["rblob"])
    if kind == "coupling":
        v_blobs = ctx.mbs(state["xb"], state["xs"], state["fs"], a_blob=state["rblob"])
        v_segs = ctx.msb(state["xs"], state["xb"], state["fb"], torch.zeros_like(state["fs"]), a_blob=state["rblob"])
        return dict(v_blobs=v_blobs, v_segs=v_segs)
    # barrier: the elastic forces of the step, and the barrier added to them
    f = state["fs"].clone()
    return dict(f_blobs=ctx.barrier(state["xs"], state["xb"], f, NSEG, scale=state["scale"]), f_segs=f)


def work(case):
    """Floating-point operations of the pair formulas (87 a pair for M_ss, 300 with the wall's images, 34 blob-blob,
    51 segment-blob, 20 to look at a barrier pair in reach), inputs read once and outputs written once."""
    kind, n, b = case["kind"], case.get("n", 0), case.get("nblob", 0)
    if kind == "segments":
        return dict(bytes=120.0 * n, flops=87.0 * n * n)
    if kind == "wall":
        return dict(bytes=120.0 * n, flops=300.0 * n * n)
    if kind == "blobs":
        return dict(bytes=72.0 * n, flops=34.0 * n * n)
    if kind == "coupling":
        return dict(bytes=168.0 * n + 96.0 * b, flops=102.0 * n * b)
    if kind == "barrier":
        return dict(bytes=120.0 * n + 48.0 * b, flops=20.0 * 30 * (n + b))
    s = case["nfil"] * NSEG
    b = case["nblob"]
    once = 87.0 * s * s + 102.0 * s * b
    if kind == "solve":
        return dict(bytes=168.0 * s + 48.0 * b, flops=once + SOLVE_ITERATIONS * 34.0 * b * b)
    return dict(bytes=8.0 * (36 * s + 9 * b), flops=STEP_EVALUATIONS * once + STEP_ITERATIONS * 34.0 * b * b +
                case["nfil"] * 2.0 * (6 * NSEG) ** 3)


# ---- the same results from plain torch in 64 bits ---------------------------------
def _rows(nt, ns, budget=1 << 22):
    step = max(1, budget // max(1, ns))
    return [(i, min(nt, i + step)) for i in range(0, nt, step)]


def _cross(ax, ay, az, bx, by, bz):
    return ay * bz - az * by, az * bx - ax * bz, ax * by - ay * bx


def _sum(*parts):
    return torch.stack([p.sum(dim=1) for p in parts], dim=1)


def _pairs(xt, xs):
    """Separations x_i - x_j, the distance (1 where it is 0) and the unit vector, (targets, sources) each."""
    d = [xt[:, c:c + 1] - xs[None, :, c] for c in range(3)]
    r = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    safe = torch.where(r > 0, r, torch.ones_like(r))
    return d, r, [c / safe for c in d]


def _exact_mss(x, f, a=1.0, mu=1.0):
    out = []
    F, T = [f[None, :, c] for c in range(3)], [f[None, :, 3 + c] for c in range(3)]
    for i, j in _rows(len(x), len(x)):
        _, r, e = _pairs(x[i:j], x)
        far = r > 2.0 * a
        s = torch.where(far, r, torch.ones_like(r))
        n6, n8 = 1.0 / (6 * math.pi * mu * a), 1.0 / (8 * math.pi * mu * a ** 3)
        i8 = 1.0 / (8 * math.pi * mu * s)
        ra = r / a
        At = torch.where(far, i8 * (1 + 2 * a * a / (3 * s * s)), n6 * (1 - 9 * ra / 32))
        Bt = torch.where(far, i8 * (1 - 2 * a * a / (s * s)), n6 * 3 * ra / 32)
        Ar = torch.where(far, -0.5 * i8 / (s * s), n8 * (1 - 27 * ra / 32 + 5 * ra ** 3 / 64))
        Br = torch.where(far, 1.5 * i8 / (s * s), n8 * (9 * ra / 32 - 3 * ra ** 3 / 64))
        C = torch.where(far, i8 / s, 0.5 * n8 * r * (1 - 3 * ra / 8))
        eF = e[0] * F[0] + e[1] * F[1] + e[2] * F[2]
        eT = e[0] * T[0] + e[1] * T[1] + e[2] * T[2]
        Te, Fe = _cross(*T, *e), _cross(*F, *e)
        out.append(_sum(*[At * F[c] + Bt * eF * e[c] + C * Te[c] for c in range(3)],
                        *[Ar * T[c] + Br * eT * e[c] + C * Fe[c] for c in range(3)]))
    return torch.cat(out)


def _exact_mbb(x, f, a=1.0, mu=1.0):
    out = []
    F = [f[None, :, c] for c in range(3)]
    for i, j in _rows(len(x), len(x)):
        _, r, e = _pairs(x[i:j], x)
        far = r > 2.0 * a
        s = torch.where(far, r, torch.ones_like(r))
        n6, i8 = 1.0 / (6 * math.pi * mu * a), 1.0 / (8 * math.pi * mu * s)
        At = torch.where(far, i8 * (1 + 2 * a * a / (3 * s * s)), n6 * (1 - 9 * r / (32 * a)))
        Bt = torch.where(far, i8 * (1 - 2 * a * a / (s * s)), n6 * 3 * r / (32 * a))
        eF = e[0] * F[0] + e[1] * F[1] + e[2] * F[2]
        out.append(_sum(*[At * F[c] + Bt * eF * e[c] for c in range(3)]))
    return torch.cat(out)


def _unequal(r, as_, ab, mu=1.0):
    """Coefficients of F, of (F.e) e and of the cross product with e, for segment radius as_ and blob radius ab."""
    far, mid = r > as_ + ab, r > abs(as_ - ab)
    s = torch.where(mid, r, torch.ones_like(r))
    i8, n6 = 1.0 / (8 * math.pi * mu * s), 1.0 / (6 * math.pi * mu * as_ * ab)
    q, d2 = as_ * as_ + ab * ab, (as_ - ab) ** 2
    t = d2 + 3 * s * s
    A = torch.where(mid, n6 * (0.5 * (as_ + ab) - t * t / (32 * s ** 3)),
                    torch.full_like(r, 1.0 / (6 * math.pi * mu * max(as_, ab))))
    A = torch.where(far, i8 * (1 + q / (3 * s * s)), A)
    B = torch.where(mid, n6 * 3 * (d2 - s * s) ** 2 / (32 * s ** 3), torch.zeros_like(r))
    B = torch.where(far, i8 * (1 - q / (s * s)), B)
    poly = (as_ - ab + s) ** 2 * (ab * ab + 2 * ab * (s + as_) - 3 * (as_ - s) ** 2) / (s * s)
    inner = r / (8 * math.pi * mu * as_ ** 3) if as_ > ab else torch.zeros_like(r)
    C = torch.where(mid, poly / (128 * math.pi * mu * ab * as_ ** 3), inner)
    return A, B, torch.where(far, i8 / s, C)


def _exact_msb(xs, xb, f, ab):
    out = []
    F = [f[None, :, c] for c in range(3)]
    for i, j in _rows(len(xs), len(xb)):
        _, r, e = _pairs(xs[i:j], xb)
        A, B, C = _unequal(r, 1.0, ab)
        eF = e[0] * F[0] + e[1] * F[1] + e[2] * F[2]
        Fe = _cross(*F, *e)
        out.append(_sum(*[A * F[c] + B * eF * e[c] for c in range(3)], *[C * Fe[c] for c in range(3)]))
    return torch.cat(out)


def _exact_mbs(xb, xs, f, ab):
    out = []
    F, T = [f[None, :, c] for c in range(3)], [f[None, :, 3 + c] for c in range(3)]
    for i, j in _rows(len(xb), len(xs)):
        _, r, e = _pairs(xb[i:j], xs)
        A, B, C = _unequal(r, 1.0, ab)
        eF = e[0] * F[0] + e[1] * F[1] + e[2] * F[2]
        Te = _cross(*T, *e)
        out.append(_sum(*[A * F[c] + B * eF * e[c] + C * Te[c] for c in range(3)]))
    return torch.cat(out)


def _exact_wall(x, f):
    """Swan and Brady's mobility above the wall z = 0 for radius and viscosity 1."""
    out = []
    k6, k8, k16 = 1 / (6 * math.pi), 1 / (8 * math.pi), 1 / (16 * math.pi)
    fx, fy, fz, tx, ty, tz = [f[None, :, c] for c in range(6)]
    for i, j in _rows(len(x), len(x), 1 << 20):
        (dx, dy, _), r, (ex, ey, ez) = _pairs(x[i:j], x)
        diag = torch.arange(i, j, device=x.device)
        r = r.clone()
        r[diag - i, diag] = 1.0
        ef, et = ex * fx + ey * fy + ez * fz, ex * tx + ey * ty + ez * tz
        s2 = 1 / (r * r)
        v = [k8 / r * ((1 + 2 * s2 / 3) * p + (1 - 2 * s2) * ef * e) for p, e in ((fx, ex), (fy, ey), (fz, ez))]
        w = [k16 * s2 / r * (3 * et * e - p) for p, e in ((tx, ex), (ty, ey), (tz, ez))]
        te, fe = _cross(tx, ty, tz, ex, ey, ez), _cross(fx, fy, fz, ex, ey, ez)
        v = [p + k8 * s2 * q for p, q in zip(v, te)]
        w = [p + k8 * s2 * q for p, q in zip(w, fe)]
        # the images
        zj = x[None, :, 2]
        zs = x[i:j, 2:3] + zj
        R = 1 / torch.sqrt(dx * dx + dy * dy + zs * zs)
        r2, r3, r4, r5 = R ** 2, R ** 3, R ** 4, R ** 5
        gx, gy, gz, h = dx * R, dy * R, zs * R, zj / zs
        gf, gt, g2 = gx * fx + gy * fy + gz * fz, gx * tx + gy * ty + gz * tz, (zs * R) ** 2
        a0 = -(0.75 * R * (1 + 2 * h * (1 - h) * g2) + 0.5 * (r3 * (1 - 3 * g2) - r5 * (1 - 5 * g2)))
        a1 = -(0.75 * R * (1 - 6 * h * (1 - h) * g2) - 1.5 * r3 * (1 - 5 * g2) + 2.5 * r5 * (1 - 7 * g2)) * gf
        a2 = gz * fz * (1.5 * h * R * (1 - 6 * (1 - h) * g2) - 3 * r3 * (1 - 5 * g2) + 5 * r5 * (2 - 7 * g2))
        a3 = (1.5 * h * R - 5 * r5) * gf
        a4 = -((3 * h * h * R + 3 * r3) * g2 + (2 - 15 * g2) * r5) * fz
        v[0] = v[0] + k6 * (a0 * fx + (a1 + a2) * gx)
        v[1] = v[1] + k6 * (a0 * fy + (a1 + a2) * gy)
        v[2] = v[2] + k6 * (a0 * fz + (a1 + a2 + a3) * gz + a4)
        a0, a1, a2, a3 = r3 * (0.375 - 2.25 * g2), -1.125 * r3 * gt, 2.25 * gz * r3 * gt, 2.25 * r3 * (gx * ty - gy * tx)
        w[0] = w[0] + k6 * (a0 * tx + a1 * gx - a3 * gy)
        w[1] = w[1] + k6 * (a0 * ty + a1 * gy + a3 * gx)
        w[2] = w[2] + k6 * (a0 * tz + a1 * gz + a2)
        a0 = 0.75 * r2
        a1 = fz * (9 * h * g2 * r2 + (1.5 - 15 * g2) * r4)
        a2 = -gz * gf * (4.5 * h * r2 - 7.5 * r4)
        a3 = -1.5 * gz * (h * r2 - r4)
        w[0] = w[0] - k6 * (a0 * (fy * gz - fz * gy) - (a1 + a2) * gy + a3 * fy)
        w[1] = w[1] - k6 * (a0 * (fz * gx - fx * gz) + (a1 + a2) * gx - a3 * fx)
        w[2] = w[2] - k6 * a0 * (fx * gy - fy * gx)
        h, gx, gy = 1 - h, -gx, -gy
        gct = gx * ty - gy * tx
        a1 = (9 * h * g2 * r2 + (1.5 - 15 * g2) * r4) * gct
        a2 = -gz * (4.5 * h * r2 - 7.5 * r4) * gct
        a3 = -1.5 * gz * (h * r2 - r4)
        v[0] = v[0] - k6 * (a0 * (tz * gy - ty * gz) + a2 * gx - a3 * ty)
        v[1] = v[1] - k6 * (a0 * (tx * gz - tz * gx) + a2 * gy + a3 * tx)
        v[2] = v[2] - k6 * (a0 * (ty * gx - tx * gy) + a2 * gz + a1)
        # a segment on itself
        h1 = 1 / x[i:j, 2]
        p = k6 - (9 * h1 - 2 * h1 ** 3 + h1 ** 5) * k6 / 16
        q = k6 - (9 * h1 - 4 * h1 ** 3 + h1 ** 5) * k6 / 8
        pr, qr = k8 - 15 * k6 / 64 * h1 ** 3, k8 - 3 * k6 / 32 * h1 ** 3
        c, g = 3 * k6 / 32 * h1 ** 4, f[i:j]
        own = [p * g[:, 0] + c * g[:, 4], p * g[:, 1] - c * g[:, 3], q * g[:, 2],
               pr * g[:, 3] - c * g[:, 1], pr * g[:, 4] + c * g[:, 0], qr * g[:, 5]]
        for m, o in zip(v + w, own):
            m[diag - i, diag] = o
        out.append(_sum(*v, *w))
    return torch.cat(out)


def _exact_barrier(xs, xb, nseg, scale):
    """Barrier forces on the segments and on the blobs (radii 1)."""
    x = torch.cat([xs, xb])
    S, out = len(xs), []
    index = torch.arange(len(x), device=x.device)
    for i, j in _rows(len(x), len(x)):
        d, r, e = _pairs(x[i:j], x)
        t, s = index[i:j, None], index[None, :]
        skip = (t < S) & (s < S) & (t // nseg == s // nseg) & ((t - s).abs() <= 1)
        inside = (r < 2.2) & ~skip & (t != s)
        c = torch.clamp(1.0 - 5.0 * (r - 2.0), max=1.0)
        c = torch.where(inside, scale * c ** 4, torch.zeros_like(r))
        out.append(_sum(*[c * k for k in e]))
    g = torch.cat(out)
    return g[:S], g[S:]


def _exact_solve(h, scale):
    """The saddle-point system of the rigid body by a dense solve."""
    xs, xb, f = h["xs"], h["refs"], h["loads"][0]
    gs, gb = _exact_barrier(xs, xb, NSEG, scale)
    f = f.clone()
    f[:, :3] += gs
    body_f = h["body_f"] + torch.cat([gb.sum(0), torch.linalg.cross(xb, gb).sum(0)])[None, :]
    n = 3 * len(xb)
    A = torch.zeros((n + 6, n + 6), dtype=F64, device=xs.device)
    d, r, e = _pairs(xb, xb)
    far = r > 2.0
    s = torch.where(far, r, torch.ones_like(r))
    At = torch.where(far, (1 + 2 / (3 * s * s)) / (8 * math.pi * s), (1 - 9 * r / 32) / (6 * math.pi))
    Bt = torch.where(far, (1 - 2 / (s * s)) / (8 * math.pi * s), 3 * r / 32 / (6 * math.pi))
    for a in range(3):
        for b in range(3):
            A[a:n:3, b:n:3] = Bt * e[a] * e[b] + (At if a == b else 0.0)
    K = torch.zeros((n, 6), dtype=F64, device=xs.device)
    for a in range(3):
        K[a::3, a] = 1.0
    x, y, z = xb[:, 0], xb[:, 1], xb[:, 2]
    K[0::3, 4], K[0::3, 5], K[1::3, 3], K[1::3, 5], K[2::3, 3], K[2::3, 4] = z, -y, -z, x, y, -x
    A[:n, n:] = -K
    A[n:, :n] = -K.T
    rhs = torch.cat([-_exact_mbs(xb, xs, f, 1.0).reshape(-1), -body_f.reshape(-1)])
    sol = torch.linalg.solve(A, rhs)
    f_blobs, v_bodies = sol[:n].reshape(-1, 3), sol[n:].reshape(1, 6)
    v_segs = _exact_mss(xs, f) + _exact_msb(xs, xb, f_blobs, 1.0)
    return dict(v_segs=v_segs, f_blobs=f_blobs, v_bodies=v_bodies, body_f=body_f)


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return None  # a whole nonlinear solve
    h = {k: torch.as_tensor(np.ascontiguousarray(v), device="cuda") for k, v in _inputs(case, seed).items()}
    if kind == "segments":
        return _exact_mss(h["xs"], h["fs"])
    if kind == "wall":
        return _exact_wall(h["xs"], h["fs"])
    if kind == "blobs":
        return _exact_mbb(h["xb"], h["fb"], case["rblob"])
    if kind == "coupling":
        return dict(v_blobs=_exact_mbs(h["xb"], h["xs"], h["fs"], case["rblob"]),
                    v_segs=_exact_msb(h["xs"], h["xb"], h["fb"], case["rblob"]))
    if kind == "barrier":
        gs, gb = _exact_barrier(h["xs"], h["xb"], NSEG, _seg_scale(case))
        f = h["fs"].clone()
        f[:, :3] += gs
        return dict(f_blobs=gb, f_segs=f)
    return _exact_solve(h, _seg_scale(case))

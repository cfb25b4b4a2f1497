"""The work that users of this framework have it do, as measurable cases.

A user builds the traction operator of a fault mesh (dense, or an H-matrix for
the large meshes), steps one simulation or an ensemble of simulations with it,
and calls the reference-shaped point functions.  ``listed()`` holds one case of
each at the sizes of this repository's benchmark and tests, from the smallest
call (64 receivers of one triangle) to the largest (the dense operator of
20,000 triangles, the H-matrix product of 100,000); ``draw()`` gives more of
the same ranges, odd and ragged sizes among them.

``exact()`` evaluates the same problem with plain torch in 64 bits: the
published angular-dislocation formulas (Nikkhoo & Walter 2015; the harmonic
free-surface term differentiated by the complex step), the aging law and the
Dormand-Prince pair.
"""
import math

import numpy as np
import torch

from pyquake3d_gb300 import _lib, gf, mesh
from pyquake3d_gb300.QDsim_gpu import STATE_FIELDS, DenseDeviceSim, initial_state
from pyquake3d_gb300.ensemble import STATE, Ensemble, PackedFixOperator, PackedOperator
from pyquake3d_gb300.hmatrix import HMatrix

MU = 32038120320.0
LAM = 32038120320.0
CS = 3464.0
V0 = 1e-6
VPL = 1e-9
ETA = MU / (2.0 * CS)
DILATANCY = {"Dilatancy coefficient": 1e-5, "Hydraulic diffusivity": 1e-6, "Actively shearing zone thickness": 1e-3,
             "Effective compressibility": 5e-11, "Constant porepressure": 5.0, "Initial porepressure": 5.0}


# ---------------------------------------------------------------------------
# cases

def listed():
    return [
        # one triangle at a few receivers through the reference's ctypes-shaped
        # call (host arrays in and out): the smallest call, all latency
        {"name": "points_64", "kind": "points", "n": 64, "half": False, "ts": 0.0},
        # the row generator of the reference's H-matrix code: one receiver, all
        # source triangles of a cluster, half space, host arrays in and out
        {"name": "sources_hs_12000", "kind": "sources", "n": 12000, "half": True, "dip": 40.0},
        # dense operator (FP64 and its FP32 copy) of the smallest configuration:
        # a planar 40 x 20 km fault of 1 km cells
        {"name": "assemble_1600", "kind": "assemble", "N": 1600, "cell": 1000.0, "rough": 0.0, "half": False,
         "dip": 90.0},
        # ... of a mid-size rough fault, the operator of the headline benchmark
        {"name": "assemble_20000", "kind": "assemble", "N": 20000, "cell": 400.0, "rough": 1e-3, "half": False,
         "dip": 90.0},
        # ... of a dipping fault that reaches the free surface (half space)
        {"name": "assemble_hs_2500", "kind": "assemble", "N": 2500, "cell": 800.0, "rough": 0.0, "half": True,
         "dip": 60.0},
        # a small simulation restarted and stepped (FP64 operator in L2: launch
        # and latency bound)
        {"name": "step_1600", "kind": "step", "N": 1600, "cell": 1000.0, "rough": 0.0, "op": "fp64", "steps": 20,
         "dila": False},
        # a mid-size simulation on its FP64 operator
        {"name": "step_20000", "kind": "step", "N": 20000, "cell": 400.0, "rough": 1e-3, "op": "fp64", "steps": 10,
         "dila": False},
        # a parameter study: 64 runs of one mesh, the arm that tracks FP64
        {"name": "batch_bf16x18_10000", "kind": "batch", "N": 10000, "cell": 1000.0, "rough": 0.0, "B": 64,
         "precision": "bf16x18", "attempt": "ff", "iters": 8},
        # a small mesh of the serving loop, 16 slots, the fast arm
        {"name": "batch_bf16x6_2000", "kind": "batch", "N": 2000, "cell": 800.0, "rough": 1e-3, "B": 16,
         "precision": "bf16x6", "attempt": "mixed", "iters": 16},
        # compression of a large mesh (partition, ACA, near field) and one product
        {"name": "hmat_build_30000", "kind": "hbuild", "N": 30000, "cell": 500.0, "rough": 1e-3, "half": False,
         "leaf": 64, "tol": 1e-4},
        # one traction product of the largest mesh
        {"name": "hmat_product_100000", "kind": "hprod", "N": 100000, "cell": 400.0, "rough": 1e-3, "leaf": 64, "B": 1},
        # a large mesh of the serving loop: 16 runs on the H-matrix
        {"name": "batch_hmat_30000", "kind": "batch", "N": 30000, "cell": 500.0, "rough": 1e-3, "B": 16,
         "precision": "hmat", "attempt": "mixed", "iters": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "sources", "assemble", "assemble", "step", "step", "batch", "batch", "hbuild", "hprod"])
    rough = rng.choice([0.0, 1e-3, 1e-3, 3e-3])
    cell = float(rng.randint(300, 1200))
    if kind == "points":
        return {"kind": kind, "n": _log(rng, 1, 100000), "half": rng.random() < 0.4, "ts": rng.choice([0.0, 0.0, 0.7])}
    if kind == "sources":
        return {"kind": kind, "n": _log(rng, 1, 40000), "half": rng.random() < 0.5, "dip": float(rng.randint(20, 75))}
    if kind == "assemble":
        if rng.random() < 0.35:
            return {"kind": kind, "N": _log(rng, 60, 2500), "cell": cell, "rough": 0.0, "half": True,
                    "dip": float(rng.randint(20, 75))}
        return {"kind": kind, "N": _log(rng, 100, 18000), "cell": cell, "rough": rough, "half": False,
                "dip": float(rng.choice([90, 90, rng.randint(20, 89)]))}
    if kind == "step":
        return {"kind": kind, "N": _log(rng, 200, 16000), "cell": cell, "rough": rough,
                "op": rng.choice(["fp64", "fp64", "fp32"]), "steps": rng.randint(5, 20), "dila": rng.random() < 0.2}
    if kind == "batch":
        p = rng.choice(["bf16x18", "bf16x18", "bf16x6", "bf16x6", "fp32", "fp64", "hmat"])
        n = {"bf16x18": (300, 9000), "bf16x6": (300, 12000), "fp32": (300, 6000), "fp64": (200, 2500),
             "hmat": (5000, 40000)}[p]
        a = {"bf16x18": ["ff", "ff", "fp64"], "bf16x6": ["mixed"], "fp32": ["mixed", "mixed", "fp64"],
             "fp64": ["fp64"], "hmat": ["mixed", "mixed", "ff"]}[p]
        return {"kind": kind, "N": _log(rng, *n), "cell": cell, "rough": 1e-3 if p == "hmat" else rough,
                "B": _log(rng, 1, 16 if p in ("fp64", "hmat") else 64), "precision": p, "attempt": rng.choice(a),
                "iters": rng.randint(2, 8)}
    if kind == "hbuild":
        return {"kind": kind, "N": _log(rng, 2000, 35000), "cell": cell, "rough": 1e-3, "half": False,
                "leaf": rng.choice([32, 64]), "tol": rng.choice([1e-4, 1e-4, 1e-5])}
    return {"kind": kind, "N": _log(rng, 3000, 90000), "cell": cell, "rough": 1e-3, "leaf": 64,
            "B": rng.choice([1, 1, 2, 3, 8, 16])}


def work(case):
    """Bytes that have to be read and written once, and the operations of the
    method at the sizes given (FP64 operations for the Green's functions: about
    500 a pair in full space, 12,000 in half space)."""
    kind = case["kind"]
    if kind in ("points", "sources"):
        return {"bytes": case["n"] * (24 if kind == "points" else 72) + case["n"] * 96.0,
                "flops": case["n"] * (12000.0 if case["half"] else 500.0)}
    N = case["N"]
    if kind == "assemble":
        return {"bytes": 72.0 * N * N, "flops": N * N * (12000.0 if case["half"] else 500.0)}
    if kind == "step":
        return {"bytes": case["steps"] * 6.0 * N * N * (8 if case["op"] == "fp64" else 4),
                "flops": case["steps"] * 12.0 * N * N}
    near = 700.0 * N * math.log2(N)   # H-matrix: about this many stored FP32 values
    if kind == "batch":
        size = {"fp64": 8, "fp32": 4, "bf16x6": 6, "bf16x18": 8, "hmat": 0}[case["precision"]]
        terms = {"fp64": 1, "fp32": 1, "bf16x6": 6, "bf16x18": 18, "hmat": 1}[case["precision"]]
        entries = near if case["precision"] == "hmat" else 6.0 * N * N
        op = 4 * near if case["precision"] == "hmat" else size * entries
        return {"bytes": case["iters"] * (op + 200.0 * N * case["B"]),
                "flops": case["iters"] * 2.0 * terms * entries * case["B"]}
    if kind == "hbuild":
        return {"bytes": 4 * near, "flops": 500.0 * near / 3}
    return {"bytes": 4 * near + 40.0 * N * case["B"], "flops": 4 * near * case["B"]}


# ---------------------------------------------------------------------------
# inputs

def _fault(case, seed, n):
    """A structured fault of n triangles (rows cut off where the grid has
    more), rough or planar, its depth direction turned to the dip angle.
    Returns (nodes, tris, length, width)."""
    rng = np.random.default_rng(seed)
    cell = case.get("cell", 500.0) * (1.0 + 0.02 * rng.random())
    nz = max(1, int(math.sqrt(n / 4.0)))
    nx = max(1, -(-n // (2 * nz)))
    L, W = nx * cell, nz * cell
    rough = case.get("rough", 0.0)
    if rough:
        nodes, tris = mesh.rough_fault(L / 1e3, W / 1e3, nx, nz, hurst=0.8, ratio=rough, seed=seed % (1 << 31))
    else:
        nodes, tris = mesh.planar_fault(L / 1e3, W / 1e3, nx, nz)
    dip = math.radians(case.get("dip", 90.0))
    if case.get("dip", 90.0) != 90.0:
        y, z = nodes[:, 1].copy(), nodes[:, 2].copy()
        nodes[:, 1] = -z * math.cos(dip) + y * math.sin(dip)
        nodes[:, 2] = z * math.sin(dip) + y * math.cos(dip)
        if rough and case.get("half"):
            nodes[:, 2] -= max(0.0, nodes[:, 2].max()) + 100.0
    return np.ascontiguousarray(nodes), np.ascontiguousarray(tris[:n]), L, W


def _points(case, seed):
    """One 1 km triangle and n receivers within 30 km of it, below the surface."""
    rng = np.random.default_rng(seed)
    P = np.array([[0.0, 0.0, -2000.0], [1000.0, 0.0, -2100.0], [300.0, -500.0, -2900.0]])
    P += rng.uniform(-100.0, 100.0, (3, 3))
    X = rng.uniform(-30e3, 30e3, (case["n"], 3))
    X[:, 2] = -np.abs(X[:, 2]) * 0.8 - 50.0
    return P, X, rng.uniform(0.5, 1.5, 2)


def _tables(case, seed, nodes, tris, L, W, B):
    _, xg = mesh.element_frames(nodes, tris)
    if B is None:
        return mesh.friction_table(xg, L, W, seed=seed % (1 << 31))
    return mesh.ensemble_tables(xg, L, W, B=B, seed=seed % (1 << 31), v_nuc=1e-3)


def _vector(B, N, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return 1e-6 * torch.randn((B, 2 * N), generator=g, dtype=torch.float64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "points":
        P, X, b = _points(case, seed)
        X = [np.ascontiguousarray(X[:, k]) for k in range(3)]
        return {"kind": kind, "args": (*X, *P, float(b[0]), float(b[1]), case["ts"], MU, LAM, case["half"])}
    if kind == "sources":
        nodes, tris, L, W = _fault(case, seed, case["n"])
        P = [np.ascontiguousarray(nodes[tris[:, k] - 1]) for k in range(3)]
        out = [np.empty((case["n"], 6)) for _ in range(2)]
        at = np.array([0.11 * L, 1500.0, -0.37 * W]) + np.random.default_rng(seed).uniform(-300.0, 300.0, 3)
        dp = [a.ctypes.data_as(_lib.c_double_p) for a in (*P, *out)]
        return {"kind": kind, "keep": (P, out), "out": out,
                "args": (*(float(v) for v in at), *dp[:3], case["n"], 1.0, 0.0, 0.0, MU, LAM, case["half"], *dp[3:])}
    nodes, tris, L, W = _fault(case, seed, case["N"])
    N, dev = case["N"], torch.device("cuda")
    if kind == "assemble":
        nodes_t, tris_t = gf.mesh_to_device(nodes, tris, dev)
        return {"kind": kind, "mesh": (nodes_t, tris_t), "half": case["half"],
                "K64": torch.empty((3 * N, 2 * N), dtype=torch.float64, device=dev),
                "K32": torch.empty((3 * N, 2 * N), dtype=torch.float32, device=dev),
                "ws": torch.empty(_lib.load().pq3d_gf_workspace_bytes(N), dtype=torch.uint8, device=dev)}
    if kind == "step":
        K64, K32 = gf.assemble_dense(nodes, tris, MU, LAM, fp32_copy=case["op"] == "fp32", device=dev)
        tab = _tables(case, seed, nodes, tris, L, W, None)
        dila = DILATANCY if case["dila"] else None
        P = np.full(N, 1e6 * DILATANCY["Initial porepressure"]) if dila else None
        sim = DenseDeviceSim(K32 if case["op"] == "fp32" else K64, initial_state(tab, V0, VPL, P=P), mu=MU, Cs=CS,
                             V0=V0, Vpl=VPL, dilatancy=dila)
        names = STATE_FIELDS + (("P", "dPdt", "Parr") if dila else ())
        return {"kind": kind, "sim": sim, "steps": case["steps"], "live": [sim.t[k] for k in names],
                "initial": [sim.t[k].clone() for k in names], "names": names}
    if kind == "batch":
        p = case["precision"]
        kw = {}
        if p == "hmat":
            K = HMatrix(nodes, tris, MU, LAM, min_size=64, mini_leaf=64, device=dev)
        else:
            K64, K32 = gf.assemble_dense(nodes, tris, MU, LAM, fp32_copy=p == "fp32", device=dev)
            if p == "bf16x6":   # K slices given, so that a run's bits do not depend on the tuner
                kw = {"nsplit": max(1, min(6, 12000 // N)), "tc_ctas": 2}
            K = {"fp64": lambda: K64, "fp32": lambda: K32, "bf16x6": lambda: PackedOperator(K64),
                 "bf16x18": lambda: PackedFixOperator(K64)}[p]()
            del K64, K32
        tabs = _tables(case, seed, nodes, tris, L, W, case["B"])
        ens = Ensemble(K, tabs, mu=MU, Cs=CS, V0=V0, Vpl=VPL, precision=p, attempt=case["attempt"], **kw)
        initial = [ens.t[k].clone() for k in STATE]
        ens.iterate(1)
        ens.capture(case["iters"])
        return {"kind": kind, "ens": ens, "live": [ens.t[k] for k in STATE], "initial": initial}
    if kind == "hbuild":
        return {"kind": kind, "mesh": (nodes, tris), "x": _vector(1, N, seed).to(dev), "leaf": case["leaf"],
                "tol": case["tol"], "half": case["half"]}
    H = HMatrix(nodes, tris, MU, LAM, min_size=case["leaf"], mini_leaf=case["leaf"], device=dev)
    B = case["B"]
    return {"kind": kind, "H": H, "x": _vector(B, N, seed).to(dev),
            "out": torch.empty((B, 3 * N), dtype=torch.float64, device=dev),
            "ws": torch.empty(H.workspace_bytes(B), dtype=torch.uint8, device=dev)}


def run(state):
    kind = state["kind"]
    if kind == "points":
        return gf.TDstressFS(*state["args"])
    if kind == "sources":
        _lib.load().TDstressEachSourceAtReceiver_C(*state["args"])
        return state["out"]
    if kind == "assemble":
        return gf.assemble_dense(*state["mesh"], MU, LAM, halfspace=state["half"], out64=state["K64"],
                                 out32=state["K32"], workspace=state["ws"])
    if kind == "step":   # the simulation from its initial state
        sim = state["sim"]
        torch._foreach_copy_(state["live"], state["initial"])
        sim.set_ctrl(dttry=1e-3, time=0.0)
        h, t, _ = sim.step(state["steps"])
        return {"h": h, "t": t, **dict(zip(state["names"], state["live"]))}
    if kind == "batch":   # the runs from their initial states
        ens = state["ens"]
        torch._foreach_copy_(state["live"], state["initial"])
        ens.set_ctrl()
        ens.prepare()
        ens.replay()
        return dict(zip(STATE, state["live"]))
    if kind == "hbuild":
        H = HMatrix(*state["mesh"], MU, LAM, min_size=state["leaf"], mini_leaf=state["leaf"], tol=state["tol"],
                    halfspace=state["half"], device=state["x"].device)
        return {"y": H.apply(state["x"]), "perm": H.perm}
    return state["H"].apply(state["x"], state["out"], state["ws"])


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch

def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def _sub(a, b):
    return tuple(x - y for x, y in zip(a, b))


def _unit(a):
    n = torch.sqrt(_dot(a, a))
    return tuple(x / n for x in a)


def _angular(x, y, z, ca, sa, bx, by, bz, nu):
    """Strain (xx, yy, zz, xy, xz, yz) of an angular dislocation in its own
    frame (Nikkhoo & Walter 2015)."""
    eta, zeta = y * ca - z * sa, y * sa + z * ca
    xx, yy, zz = x * x, y * y, z * z
    rr = xx + yy + zz
    r = torch.sqrt(rr)
    r3, rmz = rr * r, r - z
    rz, r2z2, r3z = r * rmz, rr * rmz * rmz, rr * r * rmz
    W = zeta - r
    Wr, W2 = W * r, W * W
    W2r, Wr3, W2r2 = W2 * r, W * r3, W2 * rr
    C, S = (r * ca - z) / Wr, (r * sa - y) / Wr
    k, q, p2 = 1.0 / (8.0 * math.pi * (1.0 - nu)), 1.0 / (4.0 * math.pi), 2.0 * nu + 1.0
    gx = q * (eta / r / (r - zeta) - y / r / rmz)
    gy = q * (x / r / rmz - ca * x / r / (r - zeta))
    gz = q * (sa * x / r / (r - zeta))
    fx = p2 / Wr + xx / W2r2 - xx / Wr3
    fy = 1.0 / Wr + S * S - yy / Wr3
    fz = 1.0 / Wr + C * C - zz / Wr3
    A = 1.0 / r2z2 + 1.0 / r3z
    Q3, Q4 = nu * S + xx * S / Wr + xx * y / Wr3, nu * C + xx * C / Wr + xx * z / Wr3
    yc = y * ca + z * sa
    P = sa * ca / W2 - yc / W2r + y * z / W2r2 - y * z / Wr3
    e = [-by * k * x * (fx * ca + p2 / rz - xx * A) + bz * k * x * sa * fx,
         by * gy - by * k * x * (1.0 / rz - yy * A + fy * ca) + bz * k * x * sa * fy,
         bz * gz - by * k * x * (fz * ca + z / r3) + bz * k * x * sa * fz,
         0.5 * by * gx + by * k * (xx * y * A - nu * y / rz + ca * Q3) - bz * sa * k * Q3,
         0.5 * bz * gx + by * k * (nu / r - xx / r3 + ca * Q4) - bz * sa * k * Q4,
         0.5 * (by * gz + bz * gy) - by * k * x * (y / r3 + ca * P) + bz * k * x * sa * P]
    if bx:
        e[0] = e[0] + bx * (gx + k * (eta / Wr + eta * xx / W2r2 - eta * xx / Wr3 + y / rz - xx * y * A))
        e[1] = e[1] + bx * k * (fy * eta + p2 * y / rz - yy * y * A - 2.0 * nu * ca * S)
        e[2] = e[2] + bx * k * (eta / Wr + eta * C * C - eta * zz / Wr3 + y * z / r3 + 2.0 * nu * sa * C)
        e[3] = e[3] + bx * (0.5 * gy - k * (x * yy * A - nu * x / rz - nu * x * ca / Wr + eta * x * S / Wr
                                            + eta * x * y / Wr3))
        e[4] = e[4] + bx * (0.5 * gz - k * (-x * y / r3 + nu * x * sa / Wr + eta * x * C / Wr + eta * x * z / Wr3))
        e[5] = e[5] + bx * k * (yy / r3 - nu / r - nu * ca * C + nu * sa * S + eta * sa * ca / W2 - eta * yc / W2r
                                + eta * y * z / W2r2 - eta * y * z / Wr3)
    return e


def _axes(P1, P2, P3):
    """Normal, strike and dip axes of a triangle."""
    n = _unit(_cross(_sub(P2, P1), _sub(P3, P1)))
    flat = (n[0] == 0) & (n[1] == 0)
    s = _unit((torch.where(flat, torch.zeros_like(n[0]), -n[1]), torch.where(flat, n[2], n[0]), torch.zeros_like(n[0])))
    return n, s, _cross(n, s)


def _full(X, P1, P2, P3, b, nu):
    """Strain at X of the triangles for slip b = (tensile, strike, dip)."""
    A = _axes(P1, P2, P3)
    p1, p3 = ([_dot(a, _sub(P, P2)) for a in A] for P in (P1, P3))
    e12, e13, e23 = _unit((-p1[0], -p1[1], -p1[2])), _unit(_sub(p3, p1)), _unit(p3)
    angle = (torch.acos(_dot(e12, e13)), torch.acos(-_dot(e12, e23)), torch.acos(_dot(e23, e13)))
    x, y, z = (_dot(a, _sub(X, P2)) for a in A)
    den = -p3[2] * (p1[1] - p3[1]) + p3[1] * (p1[2] - p3[2])
    a1 = (-p3[2] * (y - p3[1]) + p3[1] * (z - p3[2])) / den
    a2 = ((p1[1] - p3[1]) * (z - p3[2]) - (y - p3[1]) * (p1[2] - p3[2])) / den
    a3 = 1.0 - a1 - a2
    neg = ((a1 <= 0) & (a2 > a3) & (a3 > a1)) | ((a2 <= 0) & (a3 > a1) & (a1 > a2)) | ((a3 <= 0) & (a1 > a2) & (a2 > a3))
    sign = torch.where(neg, -1.0, 1.0).to(x.dtype)
    del a1, a2, a3, neg
    e = None
    for v, side, al, f in ((p1, e13, angle[0], -1.0), (None, e12, angle[1], 1.0), (p3, e23, angle[2], 1.0)):
        sy, sz = f * sign * side[1], f * sign * side[2]
        ty, tz = (y, z) if v is None else (y - v[1], z - v[2])
        t = _angular(x, sz * ty - sy * tz, sy * ty + sz * tz, torch.cos(al - math.pi), torch.sin(al - math.pi), b[0],
                     sz * b[1] - sy * b[2], sy * b[1] + sz * b[2], nu)
        h, d, c2, s2 = 0.5 * (t[1] + t[2]), 0.5 * (t[1] - t[2]), sz * sz - sy * sy, 2.0 * sy * sz
        u = c2 * d + s2 * t[5]
        t = (t[0], h + u, h - u, sz * t[3] + sy * t[4], sz * t[4] - sy * t[3], c2 * t[5] - s2 * d)
        e = t if e is None else tuple(p + q for p, q in zip(e, t))
    return _rotate(e, A)


def _rotate(t, A):
    """A^T T A of the symmetric T, A given by its rows."""
    T = ((t[0], t[3], t[4]), (t[3], t[1], t[5]), (t[4], t[5], t[2]))
    M = [[sum(T[i][k] * A[k][j] for k in range(3)) for j in range(3)] for i in range(3)]
    return tuple(sum(A[k][i] * M[k][j] for k in range(3)) for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)))


def _c_log(z):
    return torch.complex(torch.log(z.real), z.imag / z.real)


def _c_sqrt(z):
    r = torch.sqrt(z.real)
    return torch.complex(r, 0.5 * z.imag / r)


def _c_atan(z):
    return torch.complex(torch.atan(z.real), z.imag / (1.0 + z.real * z.real))


def _harmonic(y1, y2, y3, beta, b, nu, a):
    """Displacements of the harmonic free-surface function of an angular
    dislocation (complex arguments: the complex step)."""
    s, c = torch.sin(beta), torch.cos(beta)
    ct = c / s
    n1, n2, K = 1.0 - 2.0 * nu, 1.0 - nu, 1.0 / (4.0 * math.pi * (1.0 - nu))
    y3b = y3 + 2.0 * a
    z1b, z3b = y1 * c + y3b * s, y3b * c - y1 * s
    rb = _c_sqrt(y1 * y1 + y2 * y2 + y3b * y3b)
    rb2 = rb * rb
    rb3 = rb2 * rb
    P, Q, h, W, ar = rb + y3b, rb + z3b, y3b - a, rb * c + y3b, a / rb
    Fi = 2.0 * _c_atan(-y2 / (y1 - P / torch.tan(0.5 * beta)))
    lP, lQ = _c_log(P), _c_log(Q)
    b1, b2, b3 = (K * v for v in b)
    u1 = b1 * (-2.0 * n2 * n1 * Fi * ct * ct + n1 * y2 / P * ((n1 - ar) * ct - y1 / P * (nu + ar))
               + n1 * y2 * c * ct / Q * (c + ar) + a * y2 * h * ct / rb3
               + y2 * h / (rb * P) * (-n1 * ct + y1 / P * (2.0 * nu + ar) + a * y1 / rb2)
               + y2 * h / (rb * Q) * (c / Q * (W * (n1 * c - ar) * ct + 2.0 * n2 * (rb * s - y1) * c)
                                      - a * y3b * c * ct / rb2))
    u2 = b1 * (n1 * ((2.0 * n2 * ct * ct - nu) * lP - (2.0 * n2 * ct * ct + n1) * c * lQ)
               - n1 / P * (y1 * ct * (n1 - ar) + nu * y3b - a + y2 * y2 / P * (nu + ar))
               - n1 * z1b * ct / Q * (c + ar) - a * y1 * h * ct / rb3
               + h / P * (-2.0 * nu + (n1 * y1 * ct - a) / rb + y2 * y2 / (rb * P) * (2.0 * nu + ar) + a * y2 * y2 / rb3)
               + h / Q * (c * c - (n1 * z1b * ct + a * c) / rb + a * y3b * z1b * ct / rb3
                          - (y2 * y2 * c * c - a * z1b * ct / rb * W) / (rb * Q)))
    u3 = b1 * (2.0 * n2 * (n1 * Fi * ct + y2 / P * (2.0 * nu + ar) - y2 * c / Q * (c + ar))
               + y2 * h / rb * (2.0 * nu / P + a / rb2) + y2 * h * c / (rb * Q) * (n1 - W / Q * (c + ar) - a * y3b / rb2))
    u1 = u1 + b2 * (n1 * ((2.0 * n2 * ct * ct + nu) * lP - (2.0 * n2 * ct * ct + 1.0) * c * lQ)
                    + n1 / P * (-n1 * y1 * ct + nu * y3b - a + a * y1 * ct / rb + y1 * y1 / P * (nu + ar))
                    - n1 * ct / Q * (z1b * c - a * (rb * s - y1) / (rb * c)) - a * y1 * h * ct / rb3
                    + h / P * (2.0 * nu + (n1 * y1 * ct + a) / rb - y1 * y1 / (rb * P) * (2.0 * nu + ar)
                               - a * y1 * y1 / rb3)
                    + h * ct / Q * (-c * s + a * y1 * y3b / (rb3 * c)
                                    + (rb * s - y1) / rb * (2.0 * n2 * c - W / Q * (1.0 + a / (rb * c)))))
    u2 = u2 + b2 * (2.0 * n2 * n1 * Fi * ct * ct + n1 * y2 / P * (-(n1 - ar) * ct + y1 / P * (nu + ar))
                    - n1 * y2 * ct / Q * (1.0 + a / (rb * c)) - a * y2 * h * ct / rb3
                    + y2 * h / (rb * P) * (n1 * ct - 2.0 * nu * y1 / P - a * y1 / rb * (1.0 / rb + 1.0 / P))
                    + y2 * h * ct / (rb * Q) * (-2.0 * n2 * c + W / Q * (1.0 + a / (rb * c)) + a * y3b / (rb2 * c)))
    u3 = u3 + b2 * (-2.0 * n2 * n1 * ct * (lP - c * lQ) - 2.0 * n2 * y1 / P * (2.0 * nu + ar)
                    + 2.0 * n2 * z1b / Q * (c + ar) + h / rb * (n1 * ct - 2.0 * nu * y1 / P - a * y1 / rb2)
                    - h / Q * (c * s + W * ct / rb * (2.0 * n2 * c - W / Q)
                               + a / rb * (s - y3b * z1b / rb2 - z1b * W / (rb * Q))))
    u1 = u1 + b3 * (n1 * (y2 / P * (1.0 + ar) - y2 * c / Q * (c + ar)) - y2 * h / rb * (a / rb2 + 1.0 / P)
                    + y2 * h * c / (rb * Q) * (W / Q * (c + ar) + a * y3b / rb2))
    u2 = u2 + b3 * (n1 * (-s * lQ - y1 / P * (1.0 + ar) + z1b / Q * (c + ar)) + y1 * h / rb * (a / rb2 + 1.0 / P)
                    - h / Q * (s * (c - ar) + z1b / rb * (1.0 + a * y3b / rb2)
                               - (y2 * y2 * c * s - a * z1b / rb * W) / (rb * Q)))
    u3 = u3 + b3 * (2.0 * n2 * Fi + 2.0 * n2 * y2 * s / Q * (c + ar)
                    + y2 * h * s / (rb * Q) * (1.0 + W / Q * (c + ar) + a * y3b / rb2))
    return u1, u2, u3


def _harmonic_strain(y, beta, b, nu, a):
    tiny, J = 1e-30, []
    for k in range(3):
        yc = [torch.complex(v, torch.full_like(v, tiny if k == i else 0.0)) for i, v in enumerate(y)]
        J.append([u.imag / tiny for u in _harmonic(*yc, beta, b, nu, a)])
    return (J[0][0], J[1][1], J[2][2], 0.5 * (J[1][0] + J[0][1]), 0.5 * (J[2][0] + J[0][2]), 0.5 * (J[2][1] + J[1][2]))


def _surface_side(X, PA, PB, B, nu):
    """Free-surface correction of one side of the triangles, Burgers vector B."""
    side = _sub(PB, PA)
    hl = torch.sqrt(side[0] * side[0] + side[1] * side[1])
    beta = torch.acos(-side[2] / torch.sqrt(_dot(side, side)))
    off = (beta < 1e-4) | (math.pi - beta < 1e-4)
    hl = torch.where(off, torch.ones_like(hl), hl)
    c, s, zero = side[0] / hl, side[1] / hl, torch.zeros_like(hl)
    E = ((c, s, zero), (s, -c, zero), (zero, zero, zero - 1.0))
    yA = [_dot(e, _sub(X, PA)) for e in E]
    yB = [p - _dot(e, side) for p, e in zip(yA, E)]
    bv = [_dot(e, B) for e in E]
    f = torch.where(yA[0] >= 0.0, -1.0, 1.0).to(yA[0].dtype)     # configuration I: the mirrored frame
    bt = torch.where(yA[0] >= 0.0, math.pi - beta, beta)
    bt = torch.where(off, torch.ones_like(bt), bt)
    bv = (f * bv[0], f * bv[1], bv[2] + 0.0 * f)
    eA, eB = (_harmonic_strain((f * y[0], f * y[1], y[2] + 0.0 * f), bt, bv, nu, -P[2]) for y, P in ((yA, PA), (yB, PB)))
    d = [q - p for p, q in zip(eA, eB)]
    d[4], d[5] = f * d[4], f * d[5]
    return tuple(torch.where(off, torch.zeros_like(v), v) for v in _rotate(d, E))


def _strain(X, P, b, nu, half):
    e = _full(X, *P, b, nu)
    if not half:
        return e
    n, s, d = _axes(*P)
    B = tuple(b[0] * n[k] + b[1] * s[k] + b[2] * d[k] for k in range(3))
    top = (P[0][2] == 0) & (P[1][2] == 0) & (P[2][2] == 0)
    im = list(_full(X, *((p[0], p[1], -p[2]) for p in P), b, nu))
    im[4], im[5] = torch.where(top, -im[4], im[4]), torch.where(top, -im[5], im[5])
    e = [p + q for p, q in zip(e, im)]
    for i, j in ((0, 1), (1, 2), (2, 0)):
        e = [p + q for p, q in zip(e, _surface_side(X, P[i], P[j], B, nu))]
    return e


def _stress(e):
    tr = LAM * (e[0] + e[1] + e[2])
    return [2.0 * MU * v + (tr if k < 3 else 0.0) for k, v in enumerate(e)]


NU = LAM / (2.0 * (LAM + MU))


def _dense(nodes, tris, half):
    """The (3N, 2N) traction operator."""
    dev = torch.device("cuda")
    nodes = torch.as_tensor(nodes, device=dev)
    V = [nodes[torch.as_tensor(tris[:, k] - 1, device=dev)] for k in range(3)]
    N = len(tris)
    P = [tuple(v[:, k][None, :] for k in range(3)) for v in V]
    pc = [tuple(v[:, k] for k in range(3)) for v in V]
    g = tuple((p + q + r) / 3.0 for p, q, r in zip(*pc))
    n = _unit(_cross(_sub(pc[1], pc[0]), _sub(pc[2], pc[0])))
    flat = (n[0] == 0) & (n[1] == 0)
    one, zero = torch.ones_like(n[0]), torch.zeros_like(n[0])
    e1 = _unit((torch.where(flat, one, n[1]), torch.where(flat, zero, -n[0]), zero))
    e2 = _cross(n, e1)
    K = torch.empty((N, 3, N, 2), dtype=torch.float64, device=dev)
    step = max(1, (2_000_000 if half else 20_000_000) // N)
    for i in range(0, N, step):
        rows = slice(i, min(N, i + step))
        X, ax = tuple(v[rows, None] for v in g), [tuple(v[rows, None] for v in a) for a in (e1, e2, n)]
        for s in range(2):
            t = _stress(_strain(X, P, (0.0, 1.0 - s, float(s)), NU, half))
            u = (t[0] * ax[2][0] + t[3] * ax[2][1] + t[4] * ax[2][2], t[3] * ax[2][0] + t[1] * ax[2][1] + t[5] * ax[2][2],
                 t[4] * ax[2][0] + t[5] * ax[2][1] + t[2] * ax[2][2])
            for c in range(3):
                K[rows, c, :, s] = _dot(ax[c], u)
    return K.view(3 * N, 2 * N)


def _start(tabs):
    """The initial states of the runs, (B, N) each."""
    T = torch.as_tensor(np.asarray(tabs), dtype=torch.float64, device="cuda")
    rake, a, b, dc, f0, sig, V = (T[..., k] for k in (0, 1, 2, 3, 4, 6, 7))
    tau = sig * a * torch.asinh(V / (2.0 * V0) * torch.exp((f0 + b * math.log(V0 / VPL)) / a))
    y = {"Tno": sig, "Tt1o": tau * torch.cos(rake), "Tt2o": tau * torch.sin(rake),
         "state": torch.log(torch.sinh(tau / sig / a) * 2.0 * V0 / V) * a,
         "slipv1": V * torch.cos(rake) + 1e-16, "slipv2": V * torch.sin(rake) + 1e-16, "slipv": V, "rake": rake,
         "slip1": torch.zeros_like(V), "slip2": torch.zeros_like(V), "slip": torch.zeros_like(V), "Tt": tau,
         "fric": tau / sig}
    return y, {"a": a, "b": b, "dc": dc, "f0": f0, "shear": T[..., 8], "normal": T[..., 9], "rake0": rake}


TABLEAU = ((.2,), (3. / 40, 9. / 40), (44. / 45, -56. / 15, 32. / 9),
           (19372. / 6561, -25360. / 2187, 64448. / 6561, -212. / 729),
           (9017. / 3168, -355. / 33, -46732. / 5247, 49. / 176, -5103. / 18656),
           (35. / 384, 0., 500. / 1113, 125. / 192, -2187. / 6784, 11. / 84))
FOURTH = (5179. / 57600, 0., 7571. / 16695, 393. / 640, -92097. / 339200, 187. / 2100, 1. / 40)


def _rates(y, c, V, A1, A2, ds):
    """d(sigma, tau1, tau2, psi)/dt of the aging law with radiation damping."""
    sig, a, st = y[0] * 1e6, c["a"], y[3]
    clip = lambda v: torch.exp(torch.clamp(v, -700.0, 700.0))  # noqa: E731
    es = clip(-st / a)
    dst = c["b"] / c["dc"] * (V0 * clip((c["f0"] - st) / c["b"]) - V)
    out = []
    for t, A in ((y[1] * 1e6, A1), (y[2] * 1e6, A2)):
        p, m = clip(t / (a * sig)), clip(-t / (a * sig))
        ch, sh = 0.5 * (p + m), 0.5 * (p - m)
        dtau, dsig, dpsi = (2.0 * V0 / (a * sig) * es * ch, -2.0 * V0 * t / (a * sig * sig) * es * ch,
                            -2.0 * V0 / a * es * sh)
        out.append((c["shear"] - A - ETA * (dsig * ds + dpsi * dst)) / (1.0 + ETA * dtau) / 1e6)
    return ds / 1e6, out[0], out[1], dst


def _evolve(K, tabs, attempts=None, steps=None):
    """`attempts` attempts of every run, or the attempts that one run needs for
    `steps` accepted steps.  Returns the states and the accepted (h, t)."""
    y, c = _start(tabs)
    B, N = y["Tno"].shape
    h = torch.full((B,), 1e-3, dtype=torch.float64, device="cuda")
    time, hist, n = torch.zeros_like(h), [], 0
    while (n < attempts) if steps is None else (len(hist) < steps):
        n += 1
        v = torch.stack([y["slipv1"] - VPL * torch.cos(c["rake0"]), y["slipv2"] - VPL * torch.sin(c["rake0"])], -1)
        q = (K @ v.reshape(B, 2 * N).T).T.reshape(B, N, 3)
        f = lambda s: _rates(s, c, y["slipv"], q[..., 0], q[..., 1], q[..., 2] + c["normal"])  # noqa: E731
        y0, hc = [y[k] for k in ("Tno", "Tt1o", "Tt2o", "state")], h[:, None]
        k = [f(y0)]
        for row in TABLEAU:
            new = [y0[i] + hc * sum(w * kk[i] for w, kk in zip(row, k) if w) for i in range(4)]
            k.append(f(new))
        low = [y0[i] + hc * sum(w * kk[i] for w, kk in zip(FOURTH, k) if w) for i in range(4)]
        err = [((p - r).abs() / p).abs().amax(1) for p, r in zip(low, new)]
        e1, e2 = err[3] + 1e-10, torch.maximum(torch.maximum(err[1], err[2]), err[0]) + 1e-10
        ok = torch.maximum(e1, e2) / 1e-4 < 1.0
        want = torch.minimum(h * 0.9 * (1e-4 / e1) ** 0.2, h * 0.9 * (1e-4 / e2) ** 0.2)
        m = ok[:, None]
        sig, t1, t2, st = new
        v1, v2 = (2.0 * V0 * torch.exp(-st / c["a"]) * torch.sinh(t / sig / c["a"]) for t in (t1, t2))
        nx = {"Tno": sig, "Tt1o": t1, "Tt2o": t2, "state": st, "slipv1": v1, "slipv2": v2,
              "slipv": torch.clamp(torch.sqrt(v1 * v1 + v2 * v2), min=1e-30), "rake": torch.atan2(v2, v1),
              "slip1": y["slip1"] + v1 * hc, "slip2": y["slip2"] + v2 * hc, "Tt": torch.sqrt(t1 * t1 + t2 * t2)}
        nx["slip"] = torch.sqrt(nx["slip1"] ** 2 + nx["slip2"] ** 2)
        nx["fric"] = nx["Tt"] / sig
        y = {key: torch.where(m, nx[key], y[key]) for key in y}
        time = torch.where(ok, time + h, time)
        if steps is not None and bool(ok[0]):
            hist.append((float(h[0]), float(time[0])))
        h = torch.where(ok, torch.minimum(1.5 * h, want), torch.maximum(0.5 * h, want))
    return y, hist


def exact(case, seed):
    kind, dev = case["kind"], torch.device("cuda")
    if kind == "points":
        P, X, b = _points(case, seed)
        e = _strain(tuple(torch.as_tensor(X[:, k].copy(), device=dev) for k in range(3)),
                    [tuple(torch.as_tensor(p[k], device=dev) for k in range(3)) for p in P],
                    (case["ts"], float(b[0]), float(b[1])), NU, case["half"])
        return torch.stack(_stress(e)), torch.stack(list(e))
    if kind == "sources":
        s = prepare(case, seed)
        P = [tuple(torch.as_tensor(p[:, k].copy(), device=dev) for k in range(3)) for p in s["keep"][0]]
        e = _strain(tuple(torch.tensor(v, dtype=torch.float64, device=dev) for v in s["args"][:3]), P, (0.0, 1.0, 0.0),
                    NU, case["half"])
        return [torch.stack(_stress(e), 1), torch.stack(list(e), 1)]
    N = case["N"]
    if N > 40000 or case.get("dila"):
        return None
    nodes, tris, L, W = _fault(case, seed, N)
    K = _dense(nodes, tris, case.get("half", False))
    if kind == "assemble":
        return K, K
    if kind == "step":
        y, hist = _evolve(K, _tables(case, seed, nodes, tris, L, W, None)[None], steps=case["steps"])
        return {"h": np.array([p for p, _ in hist]), "t": np.array([p for _, p in hist]),
                **{k: y[k][0] for k in STATE_FIELDS}}
    if kind == "batch":
        y, _ = _evolve(K, _tables(case, seed, nodes, tris, L, W, case["B"]), attempts=case["iters"])
        return {k: y[k] for k in STATE}
    if kind == "hbuild":
        return {"y": (K @ _vector(1, N, seed).to(dev).T).T, "perm": None}
    return (K @ _vector(case["B"], N, seed).to(dev).T).T

"""The work a user of this framework has it do, as measurable cases.

Kinds, with the public entry point each goes through and what it stands for:
  points    TDstressFS_C of libpq3d.so on host arrays: the reference's ctypes call, made for
            single rows of a block (latency) and for post-processing grids (many receivers).
  assemble  QDsim.tree_block.master() and one product with each storage: the H-matrix of a new
            mesh, dense near field and ACA, checked by what it does to the initial deficit.
  apply     DeviceHMatrix.matvec: the six operators on one slip-rate deficit, the inner loop
            of every integrator built on the operator.
  step      QDsim.simu_forward plus the attribute reads of the reference's main loop.
  run       DeviceStepper.run and QDsim.sync_to_host: the steps between two outputs.
  vmode     VStepper.run: DP5(4) with one operator application per stage.
  ensemble  Ensemble.run: independent faults of uneven size stepped together.
  train     MLPTrainer.fit and predict: the Newton-seeding network.

Sizes: 500 to 60,000 triangles (the synthetic faults of meshgen, up to the 60k benchmark
fault), every storage precision, full and half space, absolute and relative ACA stops.
Meshes, friction and initial states come from the case and the seed alone.
"""
import ctypes
import functools
import math
import tempfile

import numpy as np
import torch

from pyquake3d_b200 import _lib, meshgen
from pyquake3d_b200.ensemble import Ensemble
from pyquake3d_b200.hmatrix import DeviceHMatrix, HStructure, pack_x
from pyquake3d_b200.mesh import get_eleVec, read_mshV2
from pyquake3d_b200.qdsim import QDsim
from pyquake3d_b200.vmode import MLPTrainer, VStepper

MU, LAM, V0, VPL = meshgen.MU, meshgen.LAM, meshgen.V0, meshgen.VPL
CS = math.sqrt(MU / meshgen.RHO)
RELTOL = 1e-4
MLP_LR = 2e-3


def listed():
    return [
        # one row of a small block through the reference's ctypes call: pure latency
        dict(name="points_64", kind="points", n=64, half=False),
        # stress on a grid of receivers near the free surface
        dict(name="points_hs_40001", kind="points", n=40001, half=True),
        # a small fault with the reference's default H-matrix settings (leaf 32, absolute stop)
        dict(name="assemble_2500", kind="assemble", n=2500, fault="planar", dip=70.0, leaf=32, tol=0.01, rel=False,
             precision="fp64", half=False),
        # the 20k thrust fault of the benchmark, mixed storage
        dict(name="assemble_20k_mixed", kind="assemble", n=20480, fault="planar", dip=30.0, leaf=64, tol=1e-4,
             rel=True, precision="mixed", half=False),
        # a half-space fault of ordinary size
        dict(name="assemble_hs_4k", kind="assemble", n=4000, fault="planar", dip=45.0, leaf=64, tol=1e-4, rel=True,
             precision="fp64", half=True),
        # the dense 2k fault: one block, FP64
        dict(name="apply_dense_1936", kind="apply", n=1936, fault="planar", dip=90.0, leaf=100000, tol=0.01,
             rel=False, precision="fp64"),
        # the 60k curved fault with its branch, mixed storage: the headline operator
        dict(name="apply_60k_mixed", kind="apply", n=60000, fault="curved", dip=90.0, leaf=64, tol=1e-5, rel=True,
             precision="mixed"),
        # one time step of the small dense fault, as the reference's main loop makes it
        dict(name="step_1936", kind="step", n=1936, fault="planar", dip=90.0, leaf=100000, tol=0.01, rel=False,
             precision="fp64"),
        # twenty steps between two outputs of a 20k fault, FP32 operator
        dict(name="run_20k_fp32", kind="run", n=20480, fault="planar", dip=30.0, leaf=64, tol=1e-4, rel=True,
             precision="fp32", steps=20),
        # V-mode on a curved fault of uneven size
        dict(name="vmode_9k_mixed", kind="vmode", n=9000, fault="curved", dip=90.0, leaf=64, tol=1e-5, rel=True,
             precision="mixed", steps=2),
        # six independent faults stepped together
        dict(name="ensemble_6", kind="ensemble", faults=6, lo=700, hi=3500, precision="mixed", steps=4),
        # one epoch of the Newton-seeding network and its predictions
        dict(name="train_65k", kind="train", n=65536, batch=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "assemble", "apply", "step", "run", "vmode", "ensemble", "train"])
    if kind == "points":
        return dict(kind=kind, n=_log(rng, 16, 40000), half=rng.random() < 0.5)
    if kind == "ensemble":
        hi = _log(rng, 800, 3500)
        return dict(kind=kind, faults=rng.randint(2, 6), lo=max(400, hi // rng.randint(2, 5)), hi=hi,
                    precision=rng.choice(["fp64", "fp32", "mixed"]), steps=rng.randint(1, 4))
    if kind == "train":
        n = _log(rng, 3000, 65536)
        return dict(kind=kind, n=n, batch=min(n, rng.choice([512, 1000, 2048, 4096])))
    fault = rng.choice(["planar", "curved"])
    c = dict(kind=kind, fault=fault, dip=90.0 if fault == "curved" else float(rng.randint(20, 90)))
    if rng.random() < 0.3:
        c.update(leaf=32, tol=0.01, rel=False)
    else:
        c.update(leaf=64, tol=rng.choice([1e-4, 1e-5]), rel=True)
    if kind == "assemble":
        c["half"] = rng.random() < 0.25
        c["n"] = _log(rng, 500, 4000 if c["half"] else 12000)
        c["precision"] = rng.choice(["fp64", "fp32", "mixed"])
    elif kind == "apply":
        c["n"] = _log(rng, 500, 24000)
        c["precision"] = rng.choice(["fp64", "fp32", "bf16", "mixed"])
    else:
        c["n"] = _log(rng, 500, 12000)
        c["precision"] = rng.choice(["fp64", "fp32", "mixed"])
        if kind != "step":
            c["steps"] = rng.randint(4, 20) if kind == "run" else rng.randint(1, 2)
    return c


# ------------------------------------------------------------------ inputs


def _mesh(case, seed):
    """Nodes (km) and triangles of a case's fault; the seed moves the interior nodes."""
    n = case["n"]
    if case["fault"] == "curved":
        return meshgen.curved_branch(n, seed=2 + seed % 1000)
    nz = max(4, int(round(math.sqrt(n / 5.0))))
    nx = max(4, int(round(n / (2.0 * nz))))
    if n == 1936:
        nx, nz = 44, 22                     # 40 x 20 km at about 1 km
    return meshgen.planar(0.6 * nx, 0.6 * nz, case["dip"], nx, nz, top=-0.5, jitter=0.1, seed=seed)


def _friction(P, T, seed):
    """The 10-column parameter rows: velocity-weakening core, 1% rate perturbation, a patch
    that slips faster."""
    xc = meshgen.centroids_km(P, T)
    half = 0.5 * (xc[:, 0].max() - xc[:, 0].min())
    zlo, zhi = xc[:, 2].min(), xc[:, 2].max()
    core = (np.abs(xc[:, 0]) < 0.8 * half) & (xc[:, 2] > zlo + 0.15 * (zhi - zlo)) & (xc[:, 2] < zhi - 0.1 * (zhi - zlo))
    c = xc[np.random.default_rng(seed).integers(len(xc))]
    cols = meshgen.friction_layout(xc, half, seed, vw_patch=lambda _: core, nuc=(c, 2.0, 1e-7))
    cols[:, 0] = 0.3 if seed % 2 else 1.2
    return cols


def _files(case, seed, folder):
    P, T = _mesh(case, seed)
    cols = _friction(P, T, seed)
    msh, para = meshgen.write_case(folder, "fault", P, T, cols, leaf=case["leaf"], tol=case["tol"], rel=case["rel"],
                                   precision=case["precision"], steps=100)
    if case.get("half"):
        with open(para) as f:
            text = f.read()
        with open(para, "w") as f:
            f.write(text.replace("Half space: False", "Half space: True"))
    return msh, para


def _sim(case, seed):
    with tempfile.TemporaryDirectory() as d:
        msh, para = _files(case, seed, d)
        nodes, tri = read_mshV2(msh)
        return QDsim(tri, nodes, para)


@functools.lru_cache(maxsize=1)
def _apply_geometry(fault, n, dip, leaf):
    P, T = _mesh(dict(fault=fault, n=n, dip=dip), 0)
    nodes = P * 1e3
    ev, xg = get_eleVec(nodes, T, False)
    return nodes, T, ev, xg, HStructure(xg, mini_leaf=leaf)


def _deficit(n, seed):
    """Slip-rate deficits (strike, dip), element order: near the plate rate, a fast patch."""
    r = np.random.default_rng(seed)
    v = VPL * (1.0 + 0.01 * r.standard_normal((2, n)))
    k = int(r.integers(n))
    v[:, k:k + max(1, n // 50)] *= 1e3
    return v[0] - VPL, v[1]


def _points(case, seed):
    """One source triangle and receivers around it (metres, all below the surface)."""
    r = np.random.default_rng(seed)
    n = case["n"]
    tri = np.array([[-400.0, 0.0, -2200.0], [500.0, 100.0, -2100.0], [50.0, 300.0, -1400.0]]) + r.normal(0, 40, (3, 3))
    x = np.stack([r.uniform(-8e3, 8e3, n), r.uniform(-8e3, 8e3, n), -r.uniform(20.0, 6e3, n)])
    return [np.ascontiguousarray(v) for v in x], [np.ascontiguousarray(p) for p in tri], r.uniform(0.5, 1.5, 3)


def _samples(n, seed):
    """Friction solves as the V-mode stepper logs them: five features and the logit of z / S
    at the root of z + kappa sinh z = S."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = torch.rand((6, n), generator=g, device="cuda", dtype=torch.float64)
    S = 5.0 + 45.0 * u[0]
    lk = -S + 6.0 * (u[1] - 0.7)
    z = torch.zeros_like(S)
    lo, hi = torch.zeros_like(S), S.clone()
    for _ in range(60):
        z = 0.5 * (lo + hi)
        f = z + 0.5 * torch.exp(lk + z) * (1.0 - torch.exp(-2.0 * z)) - S
        lo, hi = torch.where(f < 0, z, lo), torch.where(f < 0, hi, z)
    ratio = (z / S).clamp(1e-6, 1 - 1e-6)
    a, b, sig = 0.008 + 0.017 * u[2], 0.010 + 0.010 * u[3], 20.0 + 60.0 * u[4]
    f = [torch.log1p(S) / 5, lk / math.log(10.0) / 20, a * 50, b * 50, torch.log10(sig) / 2, torch.log(ratio / (1 - ratio))]
    return torch.stack(f, dim=1).float().contiguous()


def _faults(case):
    """The faults of an ensemble: sizes from lo to hi, dips from 20 to 90 degrees."""
    m = case["faults"]
    return [dict(fault="planar", n=int(case["lo"] + f * (case["hi"] - case["lo"]) / max(1, m - 1)),
                 dip=90.0 - 70.0 * f / m, leaf=64, tol=1e-5, rel=True, precision=case["precision"]) for f in range(m)]


# ------------------------------------------------------------------ state and pass


def prepare(case, seed):
    k = case["kind"]
    if k == "points":
        x, tri, b = _points(case, seed)
        n = case["n"]
        dp = ctypes.POINTER(ctypes.c_double)
        out = [np.zeros((n, 6)), np.zeros((n, 6))]
        ptrs = [a.ctypes.data_as(dp) for a in x + tri + out]
        return dict(kind=k, n=n, half=case["half"], keep=(x, tri), b=[float(v) for v in b], ptrs=ptrs, out=out,
                    lib=_lib.load())
    if k == "assemble":
        sim = _sim(case, seed)
        st = sim.tree_block.struct
        x = pack_x((sim.slipv1 - sim.slipvC * np.cos(sim.rake0))[st.perm],
                   (sim.slipv2 - sim.slipvC * np.sin(sim.rake0))[st.perm], st.n)
        x = torch.tensor(x, device="cuda")
        return dict(kind=k, sim=sim, x={torch.float64: x, torch.float32: x.float()})
    if k == "apply":
        nodes, T, ev, xg, struct = _apply_geometry(case["fault"], case["n"], case["dip"], case["leaf"])
        op = DeviceHMatrix(struct, xg, ev, nodes, T, MU, LAM, aca_tol=case["tol"], aca_rel=case["rel"])
        op.assemble(want=(case["precision"],))
        x1, x2 = _deficit(struct.n, seed)
        x = op.new_x(case["precision"])
        x.copy_(torch.tensor(pack_x(x1[struct.perm], x2[struct.perm], struct.n)))
        return dict(kind=k, op=op, x=x, precision=case["precision"])
    if k in ("step", "run"):
        sim = _sim(case, seed)
        sim._ensure_device()
        return dict(kind=k, sim=sim, dt=1e4, steps=case.get("steps", 1))
    if k == "vmode":
        sim = _sim(case, seed)
        sim.tree_block.want = (case["precision"],)
        st = VStepper(sim, sim.tree_block.op(), case["precision"])
        st.start(1e3)
        return dict(kind=k, st=st, steps=case["steps"])
    if k == "ensemble":
        sims = [_sim(c, seed + f) for f, c in enumerate(_faults(case))]
        return dict(kind=k, ens=Ensemble(sims, precision=case["precision"], want=(case["precision"],)), dt=1e4,
                    steps=case["steps"])
    if k == "train":
        return dict(kind=k, tr=MLPTrainer(seed=seed % 1000), data=_samples(case["n"], seed), batch=case["batch"])
    raise ValueError(k)


def run(s):
    k = s["kind"]
    if k == "points":
        p = s["ptrs"]
        s["lib"].TDstressFS_C(p[0], p[1], p[2], s["n"], p[3], p[4], p[5], s["b"][0], s["b"][1], s["b"][2], MU, LAM,
                              s["half"], p[6], p[7])
        return dict(stress=s["out"][0], strain=s["out"][1])
    if k == "assemble":
        op = s["sim"].tree_block.master()
        return {p: op.matvec(s["x"][P["acc"]], p) for p, P in op.plans.items()}
    if k == "apply":
        return s["op"].matvec(s["x"], s["precision"])
    if k == "step":
        sim = s["sim"]
        h, s["dt"] = sim.simu_forward(s["dt"])
        return dict(h=np.float64(h), dtnext=np.float64(s["dt"]), v1max=np.max(np.abs(sim.slipv1)),
                    v2max=np.max(np.abs(sim.slipv2)), slipv=sim.slipv, Tt=sim.Tt)
    if k == "run":
        sim = s["sim"]
        hist = sim._ensure_device().run(s["steps"], s["dt"])
        s["dt"] = float(hist[-1, 1])
        sim.sync_to_host()
        return dict(h=hist[:, 0], slipv=sim.slipv, Tt=sim.Tt, Tno=sim.Tno, state=sim.state, slip=sim.slip)
    if k == "vmode":
        st = s["st"]
        c = st.run(s["steps"], chunk=s["steps"])
        return dict(time=c[2], y=st.y0, V=st.V)
    if k == "ensemble":
        e = s["ens"]
        hist = e.run(s["steps"], s["dt"])
        s["dt"] = hist[-1, :, 1].copy()
        return dict(h=hist[:, :, 0], slipv=[e.get("slipv", f) for f in range(e.M)],
                    Tt=[e.get("Tt", f) for f in range(e.M)])
    tr = s["tr"]
    tr.fit(s["data"], epochs=1, batch=s["batch"], lr=MLP_LR)
    return dict(P=tr.P, Y=tr.predict(s["data"]))


# Mean ACA terms of a block (both slips) per stop, for the size estimates of work().
_TERMS = {(0.01, False): 47.0, (1e-4, True): 26.0, (1e-5, True): 52.0}
_PAIR_FLOPS = 1600.0             # both slips of one full-space pair


def _entries(case):
    """(dense entries, sum of (m + n) over the low-rank blocks) of a case's block tree."""
    P, T = _mesh(case, 0)
    xg = meshgen.centroids_km(P, T) * 1e3
    st = HStructure(xg, mini_leaf=case["leaf"]).stats()
    return st["n"], st["dense_entries"], st["aca_m_plus_n"]


def work(case):
    k = case["kind"]
    if k == "points":
        return dict(bytes=case["n"] * (3 + 12) * 8.0, flops=case["n"] * (8.0 if case["half"] else 1.0) * _PAIR_FLOPS)
    if k == "train":
        n = case["n"] // case["batch"] * case["batch"]
        return dict(bytes=24.0 * n, flops=2.0 * 4480 * 3 * n + 2.0 * 4480 * case["n"])
    if k == "ensemble":
        w = [work(dict(c, kind="run", steps=case["steps"])) for c in _faults(case)]
        return {key: sum(v[key] for v in w) for key in ("bytes", "flops")}
    n, dense, mn = _entries(case)
    terms = _TERMS[case["tol"], case["rel"]]
    if k == "assemble":
        out = (8.0 if case["precision"] != "fp32" else 12.0) + (4.0 if case["precision"] == "mixed" else 0.0)
        return dict(bytes=out * (6.0 * dense + 3 * terms * mn),
                    flops=(8.0 if case["half"] else 1.0) * (_PAIR_FLOPS * dense + 0.6 * _PAIR_FLOPS * terms * mn))
    size = {"fp64": (8.0, 8.0), "fp32": (4.0, 4.0), "bf16": (4.0, 2.0), "mixed": (4.0, 2.2)}[case["precision"]]
    apply = size[0] * 6 * dense + size[1] * 3 * terms * mn + 2 * n * size[0] + 24.0 * n
    flops = 2.0 * (6 * dense + 3 * terms * mn)
    per = {"apply": 1, "step": 1, "run": case.get("steps", 1), "vmode": 6 * case.get("steps", 1)}[k]
    return dict(bytes=per * (apply + (0 if k == "apply" else 300.0 * n)), flops=per * (flops + (0 if k == "apply" else 1e3 * n)))


# ------------------------------------------------------------------ the same in 64 bits


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _angular(x, y, z, ca, sa, b, nu):
    """Strain (xx, yy, zz, xy, xz, yz) of an angular dislocation with Burgers vector b
    (Nikkhoo & Walter 2015, appendix; the vertical side along z, the other at angle alpha)."""
    bx, by, bz = b
    eta, zeta = y * ca - z * sa, y * sa + z * ca
    x2, y2, z2 = x * x, y * y, z * z
    r2 = x2 + y2 + z2
    r = r2.sqrt()
    r3 = r2 * r
    rz = r * (r - z)
    r2z2, r3z = rz * rz, r3 * (r - z)
    W = zeta - r
    W2 = W * W
    Wr, W2r, Wr3, W2r2 = W * r, W2 * r, W * r3, W2 * r2
    C, S = (r * ca - z) / Wr, (r * sa - y) / Wr
    fx = (eta / r / (r - zeta) - y / r / (r - z)) / 4 / math.pi
    fy = (x / r / (r - z) - ca * x / r / (r - zeta)) / 4 / math.pi
    fz = (sa * x / r / (r - zeta)) / 4 / math.pi
    k = 1 / (8 * math.pi * (1 - nu))
    n1 = 2 * nu + 1
    exx = bx * fx + bx * k * (eta / Wr + eta * x2 / W2r2 - eta * x2 / Wr3 + y / rz - x2 * y / r2z2 - x2 * y / r3z) \
        - by * x * k * ((n1 / Wr + x2 / W2r2 - x2 / Wr3) * ca + n1 / rz - x2 / r2z2 - x2 / r3z) \
        + bz * x * sa * k * (n1 / Wr + x2 / W2r2 - x2 / Wr3)
    eyy = by * fy + bx * k * ((1 / Wr + S * S - y2 / Wr3) * eta + n1 * y / rz - y2 * y / r2z2 - y2 * y / r3z
                              - 2 * nu * ca * S) \
        - by * x * k * (1 / rz - y2 / r2z2 - y2 / r3z + (1 / Wr + S * S - y2 / Wr3) * ca) \
        + bz * x * sa * k * (1 / Wr + S * S - y2 / Wr3)
    ezz = bz * fz + bx * k * (eta / Wr + eta * C * C - eta * z2 / Wr3 + y * z / r3 + 2 * nu * sa * C) \
        - by * x * k * ((1 / Wr + C * C - z2 / Wr3) * ca + z / r3) \
        + bz * x * sa * k * (1 / Wr + C * C - z2 / Wr3)
    exy = bx * fy / 2 + by * fx / 2 \
        - bx * k * (x * y2 / r2z2 - nu * x / rz + x * y2 / r3z - nu * x * ca / Wr + eta * x * S / Wr + eta * x * y / Wr3) \
        + by * k * (x2 * y / r2z2 - nu * y / rz + x2 * y / r3z + nu * ca * S + x2 * y * ca / Wr3 + x2 * ca * S / Wr) \
        - bz * sa * k * (nu * S + x2 * S / Wr + x2 * y / Wr3)
    exz = bx * fz / 2 + bz * fx / 2 \
        - bx * k * (-x * y / r3 + nu * x * sa / Wr + eta * x * C / Wr + eta * x * z / Wr3) \
        + by * k * (-x2 / r3 + nu / r + nu * ca * C + x2 * z * ca / Wr3 + x2 * ca * C / Wr) \
        - bz * sa * k * (nu * C + x2 * C / Wr + x2 * z / Wr3)
    q = y * ca + z * sa
    eyz = by * fz / 2 + bz * fy / 2 \
        + bx * k * (y2 / r3 - nu / r - nu * ca * C + nu * sa * S + eta * sa * ca / W2 - eta * q / W2r
                    + eta * y * z / W2r2 - eta * y * z / Wr3) \
        - by * x * k * (y / r3 + sa * ca * ca / W2 - ca * q / W2r + y * z * ca / W2r2 - y * z * ca / Wr3) \
        - bz * x * sa * k * (y * z / Wr3 - sa * ca / W2 + q / W2r - y * z / W2r2)
    return exx, eyy, ezz, exy, exz, eyz


def _tensor(e):
    return torch.stack([torch.stack([e[0], e[3], e[4]], -1), torch.stack([e[3], e[1], e[5]], -1),
                        torch.stack([e[4], e[5], e[2]], -1)], -2)


def _td_strain(obs, tri, burgers):
    """Strain tensors (..., 3, 3) at obs (R, 3) of triangles tri (C, 3, 3), full space, as
    (R, C): three angular dislocations per triangle, the configuration by barycentric signs.
    burgers: (tensile, strike, dip) components, numbers."""
    nu = LAM / (2 * (LAM + MU))
    P1, P2, P3 = tri[:, 0], tri[:, 1], tri[:, 2]
    vn = _unit(torch.linalg.cross(P2 - P1, P3 - P1))
    vs = _unit(torch.stack([-vn[:, 1], vn[:, 0], torch.zeros_like(vn[:, 0])], 1))
    vd = torch.linalg.cross(vn, vs)
    A = torch.stack([vn, vs, vd], 1)                                    # rows: the triangle's axes
    X = torch.einsum("cij,rcj->rci", A, obs[:, None] - P2[None])
    p1, p3 = torch.einsum("cij,cj->ci", A, P1 - P2), torch.einsum("cij,cj->ci", A, P3 - P2)
    p2 = torch.zeros_like(p1)
    e12, e13, e23 = _unit(p2 - p1), _unit(p3 - p1), _unit(p3 - p2)
    angles = [torch.acos((u * v).sum(1)) for u, v in ((e12, e13), (-e12, e23), (e23, e13))]
    x, y, z = X[..., 0], X[..., 1], X[..., 2]
    den = (p2[:, 2] - p3[:, 2]) * (p1[:, 1] - p3[:, 1]) + (p3[:, 1] - p2[:, 1]) * (p1[:, 2] - p3[:, 2])
    a = ((p2[:, 2] - p3[:, 2]) * (y - p3[:, 1]) + (p3[:, 1] - p2[:, 1]) * (z - p3[:, 2])) / den
    b = ((p3[:, 2] - p1[:, 2]) * (y - p3[:, 1]) + (p1[:, 1] - p3[:, 1]) * (z - p3[:, 2])) / den
    c = 1 - a - b
    neg = ((a <= 0) & (b > c) & (c > a)) | ((b <= 0) & (c > a) & (a > b)) | ((c <= 0) & (a > b) & (b > c))
    sg = torch.where(neg, -1.0, 1.0).to(x.dtype)
    bn, bs, bd = burgers
    total = None
    for ang, pos, side in zip(angles, (p1, p2, p3), (-e13, e12, e23)):
        s1, s2 = sg * side[:, 1], sg * side[:, 2]
        yy, zz = y - pos[:, 1], z - pos[:, 2]
        # rotation about x that brings the side onto the z axis
        y1, z1 = s2 * yy - s1 * zz, s1 * yy + s2 * zz
        by, bz = s2 * bs - s1 * bd, s1 * bs + s2 * bd
        t = ang - math.pi
        e = _angular(x, y1, z1, torch.cos(t), torch.sin(t), (bn, by, bz), nu)
        # back: R^T e R with R = [[1, 0, 0], [0, s2, -s1], [0, s1, s2]]
        exx, eyy, ezz, exy, exz, eyz = e
        f = [exx, s2 * s2 * eyy + 2 * s1 * s2 * eyz + s1 * s1 * ezz, s1 * s1 * eyy - 2 * s1 * s2 * eyz + s2 * s2 * ezz,
             s2 * exy + s1 * exz, -s1 * exy + s2 * exz,
             -s1 * s2 * eyy + (s2 * s2 - s1 * s1) * eyz + s1 * s2 * ezz]
        total = f if total is None else [u + v for u, v in zip(total, f)]
    return torch.einsum("cki,rckl,clj->rcij", A, _tensor(total), A)


def _hooke(e):
    tr = e.diagonal(dim1=-2, dim2=-1).sum(-1)
    return 2 * MU * e + LAM * tr[..., None, None] * torch.eye(3, dtype=e.dtype, device=e.device)


def _frames(nodes, tri):
    """Centroids, element axes (strike, dip, normal; normals along (b - a) x (c - a))."""
    v = nodes[tri - 1]
    n = _unit(torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]))
    e1 = _unit(torch.stack([n[:, 1], -n[:, 0], torch.zeros_like(n[:, 0])], 1))
    return v.mean(1), torch.stack([e1, torch.linalg.cross(n, e1), n], 1), v


def _operator(P, T):
    """x (2, n) -> (3, n): shear along strike and dip and normal traction at every element of
    the fault, each pair from the full-space solution.  Kept as one dense array when it fits."""
    nodes, tri = torch.tensor(P * 1e3, device="cuda"), torch.tensor(T, device="cuda")
    xg, frame, v = _frames(nodes, tri)
    n = len(tri)

    def rows(r0, r1):
        K = torch.empty((2, 3, r1 - r0, n), dtype=torch.float64, device="cuda")
        for s in range(2):
            sig = _hooke(_td_strain(xg[r0:r1], v, (0.0, 1.0 - s, float(s))))
            t = torch.einsum("rcij,rj->rci", sig, frame[r0:r1, 2])
            K[s] = torch.einsum("rkj,rcj->krc", frame[r0:r1], t)
        return K
    step = max(1, 2_000_000 // n)
    cuts = [(r, min(n, r + step)) for r in range(0, n, step)]
    if n <= 24000:
        K = torch.empty((2, 3, n, n), dtype=torch.float64, device="cuda")
        for r0, r1 in cuts:
            K[:, :, r0:r1] = rows(r0, r1)
        return lambda x: torch.stack([K[0, c] @ x[0] + K[1, c] @ x[1] for c in range(3)])

    def apply(x):
        return torch.cat([torch.stack([k[0, c] @ x[0] + k[1, c] @ x[1] for c in range(3)])
                          for k in (rows(r0, r1) for r0, r1 in cuts)], 1)
    return apply


# Dormand-Prince 5(4)
_A = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, -46732 / 5247, 49 / 176, -5103 / 18656],
      [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_B4 = [5179 / 57600, 0.0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40]


class _Fault:
    """Initial state of a parameter file's rows and the operator, element order, 64 bits."""

    def __init__(self, P, T, cols):
        t = torch.tensor(cols, device="cuda")
        self.rake, self.a, self.b, self.dc, self.f0 = t[:, 0], t[:, 1], t[:, 2], t[:, 3], t[:, 4]
        self.Tn, V, self.shear, self.normal = t[:, 6], t[:, 7], t[:, 8], t[:, 9]
        c, s = torch.cos(self.rake), torch.sin(self.rake)
        self.c, self.s = c, s
        self.V, self.V1, self.V2 = V.clone(), V * c + 1e-16, V * s + 1e-16
        Tt = self.Tn * self.a * torch.asinh(V / (2 * V0) * torch.exp((self.f0 + self.b * math.log(V0 / VPL)) / self.a))
        self.T1, self.T2 = Tt * c, Tt * s
        self.psi = torch.log(torch.sinh(Tt / self.Tn / self.a) * 2 * V0 / V) * self.a
        self.slip1, self.slip2 = torch.zeros_like(V), torch.zeros_like(V)
        self.eta = MU / (2 * CS)
        self.K = _operator(P, T)

    def rates(self, L, y):
        Tn, T1, T2, psi = (1e6 * y[0], 1e6 * y[1], 1e6 * y[2], y[3])
        dsig = L[2] + self.normal
        dpsi = self.b / self.dc * (V0 * torch.exp(((self.f0 - psi) / self.b).clamp(-700, 700)) - self.V)
        out = [dsig * 1e-6]
        for T, A in ((T1, L[0]), (T2, L[1])):
            z = T / (self.a * Tn)
            ch, sh = 2 * V0 * torch.exp(-psi / self.a) * torch.cosh(z), 2 * V0 * torch.exp(-psi / self.a) * torch.sinh(z)
            dtau, dsg, dst = ch / (self.a * Tn), -ch * T / (self.a * Tn * Tn), -sh / self.a
            out.append((-A + self.shear - self.eta * (dsg * dsig + dst * dpsi)) / (1 + self.eta * dtau) * 1e-6)
        return torch.stack(out + [dpsi])

    def step(self, h):
        """One step of the frozen-load DP5(4) scheme with its controller; (h taken, next h)."""
        L = self.K(torch.stack([self.V1 - VPL * self.c, self.V2 - VPL * self.s]))
        y0 = torch.stack([self.Tn, self.T1, self.T2, self.psi])
        while True:
            k = []
            for row in _A:
                k.append(self.rates(L, y0 + h * sum((w * v for w, v in zip(row, k)), torch.zeros_like(y0))))
            y5 = y0 + h * sum(w * v for w, v in zip(_A[6], k))
            y4 = y0 + h * sum(w * v for w, v in zip(_B4, k))
            e = ((y4 - y5).abs() / y4.abs()).amax(1).tolist()
            R1, R2 = e[3] + 1e-10, max(e[:3]) + 1e-10
            h1, h2 = 0.9 * h * (RELTOL / R1) ** 0.2, 0.9 * h * (RELTOL / R2) ** 0.2
            if max(R1, R2) < RELTOL:
                break
            h = max(0.5 * h, min(h1, h2))
        self.Tn, self.T1, self.T2, self.psi = y5
        ex = 2 * V0 * torch.exp(-self.psi / self.a)
        self.V1, self.V2 = ex * torch.sinh(self.T1 / self.Tn / self.a), ex * torch.sinh(self.T2 / self.Tn / self.a)
        self.V = torch.hypot(self.V1, self.V2).clamp(min=1e-30)
        self.slip1, self.slip2 = self.slip1 + h * self.V1, self.slip2 + h * self.V2
        return h, min(h1, h2, 1.5 * h)

    def vmode(self, h, steps):
        """DP5(4) on (slip, state) with the slip rates from the damped friction law: `steps`
        attempts at a time until `steps` or more are accepted; (time, slip and state, rates)."""
        tq = [1e6 * self.T1 + self.eta * self.V1, 1e6 * self.T2 + self.eta * self.V2]
        sig0 = 1e6 * self.Tn
        y, t, done = torch.stack([self.slip1, self.slip2, self.psi]), 0.0, 0

        def f(t, y):
            d = torch.stack([y[0] - VPL * self.c * t, y[1] - VPL * self.s * t])
            L = self.K(d)
            sig = sig0 + L[2] + self.normal * t
            V = []
            for q, A in zip(tq, L):
                T = q - A + self.shear * t
                S = T.abs() / (self.a * sig)
                lk = torch.log(2 * V0 * self.eta / (self.a * sig)) - y[2] / self.a
                z = S.clone()
                for _ in range(60):
                    g, u = torch.exp(lk + z), torch.exp(-2 * z)
                    z = torch.minimum((z - (z + 0.5 * g * (1 - u) - S) / (1 + 0.5 * g * (1 + u))).clamp(min=0), S)
                V.append(torch.sign(T) * V0 * torch.exp(z - y[2] / self.a) * (1 - torch.exp(-2 * z)))
            dpsi = self.b / self.dc * (V0 * torch.exp(((self.f0 - y[2]) / self.b).clamp(-700, 700)) - torch.hypot(*V))
            return torch.stack(V + [dpsi])
        k1 = f(0.0, y)
        tried = 0
        while done < steps or tried % steps:
            tried += 1
            k = [k1]
            for row, c in zip(_A[1:], (0.2, 0.3, 0.8, 8 / 9, 1.0, 1.0)):
                k.append(f(t + c * h, y + h * sum(w * v for w, v in zip(row, k))))
            y5 = y + h * sum(w * v for w, v in zip(_A[6], k))
            e = (y5 - y - h * sum(w * v for w, v in zip(_B4, k))).abs()
            scale = torch.stack([y5[0].abs() + 1e-9, y5[1].abs() + 1e-9, y5[2].abs()])
            E = float((e / scale).max()) / RELTOL
            hn = 0.9 * h * E ** -0.2 if E > 0 else 1.5 * h
            if E < 1:
                y, t, k1, done, h = y5, t + h, k[6], done + 1, min(hn, 1.5 * h)
            else:
                h = max(0.5 * h, hn)
        return t, y, k[6][:2]


def _exact_train(case, seed):
    """The same epoch of Adam steps in 64 bits from the same start and sample order."""
    data = _samples(case["n"], seed).double()
    r = np.random.default_rng(seed % 1000)
    W = [r.normal(0, 1 / np.sqrt(5), (64, 5)), np.zeros(64), r.normal(0, 1 / 8.0, (64, 64)), np.zeros(64),
         r.normal(0, 1 / 8.0, (1, 64)), np.zeros(1)]
    W = [torch.tensor(w, device="cuda").float().double().requires_grad_() for w in W]
    m, v = [torch.zeros_like(w) for w in W], [torch.zeros_like(w) for w in W]

    def net(X):
        h = torch.tanh(X @ W[0].T + W[1])
        h = torch.tanh(h @ W[2].T + W[3])
        return (h @ W[4].T + W[5])[:, 0]
    g = torch.Generator(device="cuda")
    g.manual_seed(0)
    order = torch.randperm(case["n"], device="cuda", generator=g)
    B = case["batch"]
    for t, s in enumerate(range(0, case["n"] - B + 1, B), 1):
        d = data[order[s:s + B]]
        grads = torch.autograd.grad(0.5 * ((net(d[:, :5]) - d[:, 5]) ** 2).mean(), W)
        with torch.no_grad():
            for w, a, q, gr in zip(W, m, v, grads):
                a.mul_(0.9).add_(0.1 * gr)
                q.mul_(0.999).add_(0.001 * gr * gr)
                w -= MLP_LR * (a / (1 - 0.9 ** t)) / ((q / (1 - 0.999 ** t)).sqrt() + 1e-8)
    with torch.no_grad():
        return dict(P=torch.cat([w.reshape(-1) for w in W]), Y=net(data[:, :5]))


def exact(case, seed):
    k = case["kind"]
    if case.get("half"):
        return None                     # the free-surface terms have no short form
    if k == "points":
        x, tri, b = _points(case, seed)
        obs = torch.tensor(np.stack(x, 1), device="cuda")
        e = _td_strain(obs, torch.tensor(np.stack(tri), device="cuda")[None], (b[2], b[0], b[1]))[:, 0]
        pick = lambda t: torch.stack([t[:, 0, 0], t[:, 1, 1], t[:, 2, 2], t[:, 0, 1], t[:, 0, 2], t[:, 1, 2]], 1)
        return dict(stress=pick(_hooke(e)), strain=pick(e))
    if k == "apply":
        P, T = _mesh(case, 0)
        x1, x2 = _deficit(len(T), seed)
        y = _operator(P, T)(torch.tensor(np.stack([x1, x2]), device="cuda")).T
        return y[_tree_order(P, T)]
    if k in ("step", "run", "vmode"):
        P, T = _mesh(case, seed)
        f = _Fault(P, T, _friction(P, T, seed))
        if k == "vmode":
            t, y, V = f.vmode(1e3, case["steps"])
            order = _tree_order(P, T)
            return dict(time=torch.tensor(t, dtype=torch.float64), y=y[:, order].reshape(-1), V=V[:, order].reshape(-1))
        h, hs = 1e4, []
        for _ in range(case.get("steps", 1)):
            took, h = f.step(h)
            hs.append(took)
        Tt = torch.hypot(f.T1, f.T2)
        if k == "step":
            return dict(h=np.float64(hs[0]), dtnext=np.float64(h), v1max=f.V1.abs().max(), v2max=f.V2.abs().max(),
                        slipv=f.V, Tt=Tt)
        return dict(h=np.array(hs), slipv=f.V, Tt=Tt, Tno=f.Tn, state=f.psi, slip=torch.hypot(f.slip1, f.slip2))
    if k == "ensemble":
        slipv, Tt, took = [], [], []
        for i, c in enumerate(_faults(case)):
            P, T = _mesh(c, seed + i)
            f = _Fault(P, T, _friction(P, T, seed + i))
            h, hs = 1e4, []
            for _ in range(case["steps"]):
                t, h = f.step(h)
                hs.append(t)
            took.append(hs)
            slipv.append(f.V)
            Tt.append(torch.hypot(f.T1, f.T2))
        return dict(h=np.array(took).T.copy(), slipv=slipv, Tt=Tt)
    if k == "train":
        return _exact_train(case, seed)
    P, T = _mesh(case, seed)
    f = _Fault(P, T, _friction(P, T, seed))
    y = f.K(torch.stack([f.V1 - VPL * f.c, f.V2 - VPL * f.s])).T[_tree_order(P, T)]
    return {p: y for p in {"fp64", case["precision"]}}


def _tree_order(P, T, leaf=16):
    """Elements in cluster-tree order: bisection of the longest axis of the bounding box at
    its midpoint, left part first, down to `leaf` elements."""
    v = [(P * 1e3)[T[:, k] - 1] for k in range(3)]
    xg = (v[0] + v[1] + v[2]) / 3.0
    out, stack = [], [np.arange(len(xg))]
    while stack:
        idx = stack.pop()
        p = xg[idx]
        lo, hi = p.min(0), p.max(0)
        j = int(np.argmax(hi - lo))
        left = p[:, j] <= (lo[j] + hi[j]) / 2
        if len(idx) <= leaf or left.all() or not left.any():
            out.append(idx)
        else:
            stack += [idx[~left], idx[left]]
    return torch.tensor(np.concatenate(out), device="cuda")

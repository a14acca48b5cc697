"""The solver's work, as its users run it, in sizes small enough to repeat.

Every time-loop case is a stretch of a run in progress: a model is built with
the mesh generator, a seeded wavefield is put into the solver as a restart
would (``Solver.set_state``), and one pass advances it by whole snapshot
intervals and reads every snapshot back through ``Solver.run``, as a run that
collects strain Green's functions does.  The cases cover both precisions, the
polynomial orders 2 to 5, one to six wavefields, C-PML and the legacy damping
layer, homogeneous, layered and deformed meshes from under a thousand cells
to eighty thousand, several models in one solver, the restart read-out,
and the element residual on the caller's device buffers.

``exact`` states the same time loop (central differences, cell by cell C-PML
memory) in plain 64-bit torch.
"""

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gf-only-sem_b200"))

import gfb  # noqa: E402
from gfb import mesh, workloads  # noqa: E402

STRIDE = 10  # steps between snapshots, as in the named workloads


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def _loop(kind, nx, ny, nz, order, precision, dirs, pml, passes, **more):
    """A time-loop case: mesh kind and cells per axis, polynomial order,
    precision, force directions (a text of x, y, z), absorbing cells per face,
    snapshot intervals per pass."""
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "order": order, "precision": precision, "dirs": dirs,
         "pml": pml, "cpml": True, "tile": 8, "intervals": passes, "sources": 1, "state": False}
    c.update(more)
    return c


def listed():
    return [
        # the smallest run kept on disk between restarts: a ragged box, one
        # force direction in FP64 (what the executable runs by default), the
        # full state read out as for a restart file
        dict(_loop("layered", 11, 9, 7, 4, "fp64", "y", 1, 5, tile=5, state=True), name="restart_small_fp64"),
        # the 20 x 20 x 10 halfspace that the CPU oracle runs in full: small
        # enough for launches and gaps to count
        dict(_loop("halfspace", 20, 20, 10, 4, "fp32", "xyz", 3, 4), name="halfspace_small_fp32"),
        # an ordinary flat-layered model, three force directions batched
        dict(_loop("layered", 40, 40, 20, 4, "fp32", "xyz", 4, 2, tile=12), name="layered_fp32"),
        # the same model in FP64, one direction: a parity run
        dict(_loop("layered", 40, 40, 20, 4, "fp64", "z", 4, 1, tile=12), name="layered_fp64"),
        # the production shape: deformed mesh, topography, random medium
        dict(_loop("deformed", 52, 54, 27, 4, "fp32", "xyz", 5, 1, tile=16), name="deformed_large_fp32"),
        # the other polynomial orders, ragged boxes, fewer wavefields
        dict(_loop("layered", 37, 29, 23, 2, "fp32", "xyz", 3, 2), name="order2_fp32"),
        dict(_loop("layered", 30, 31, 17, 3, "fp32", "xy", 3, 2), name="order3_fp32"),
        dict(_loop("deformed", 22, 21, 13, 5, "fp32", "xyz", 2, 2), name="order5_fp32"),
        # the legacy damping layer instead of C-PML, three directions in FP64
        dict(_loop("layered", 24, 25, 12, 4, "fp64", "xyz", 3, 1, cpml=False), name="damping_fp64"),
        # two source positions times three directions in one solver
        dict(_loop("deformed", 32, 32, 16, 4, "fp32", "xyz", 5, 1, sources=2), name="two_sources_fp32"),
        # several models of uneven size advanced together
        dict(_batch(6, 7, 4), name="batch_fp32"),
        # K_e u of one block of cells on the caller's device buffers
        {"kind": "element", "order": 4, "cells": 600, "name": "element_residual"},
    ]


def _batch(models, n0, passes):
    """``models`` layered models of n0, n0+2, ... cells along x."""
    return {"kind": "batch", "models": models, "n0": n0, "order": 4, "precision": "fp32", "dirs": "xyz", "pml": 2,
            "cpml": True, "tile": 3, "intervals": passes, "sources": 1, "state": False}


def draw(rng):
    kind = rng.choice(["fp32", "fp32", "fp32", "fp64", "fp64", "orders", "batch", "sources", "element"])
    if kind == "element":
        order = rng.choice([2, 3, 4, 4, 5])
        most = {2: 3106, 3: 1310, 4: 671, 5: 388}[order]
        return {"kind": "element", "order": order, "cells": int(math.exp(rng.uniform(0.0, math.log(most))))}
    if kind == "batch":
        return _batch(rng.randint(2, 7), rng.randint(5, 9), rng.randint(2, 4))
    lo, hi = math.log(400.0), math.log({"fp32": 75000.0, "fp64": 34000.0, "orders": 12000.0, "sources": 18000.0}[kind])
    n = math.exp(rng.uniform(lo, hi)) ** (1.0 / 3.0)
    nx, ny = (max(6, int(n * rng.uniform(1.0, 1.5))) for _ in range(2))
    nz = max(5, int(n ** 3 / (nx * ny)))
    pml = rng.randint(1, max(1, min(4, (min(nx, ny) - 3) // 3)))
    tile = min(8, nx - 2 * pml - 1, ny - 2 * pml - 1)
    medium = rng.choice(["halfspace", "layered", "deformed"])
    dirs = rng.choice(["x", "z", "yz", "xyz", "xyz", "xyz"])
    few = nx * ny * nz < 8000
    args = dict(tile=tile, passes=rng.randint(2, 4) if few else rng.randint(1, 2))
    if kind == "orders":
        return _loop(medium, nx, ny, nz, rng.choice([2, 3, 5]), rng.choice(["fp32", "fp32", "fp64"]), dirs, pml, **args)
    if kind == "sources":
        return _loop(medium, nx, ny, nz, 4, "fp32", "xyz", pml, sources=rng.choice([2, 2, 3]), **args)
    if kind == "fp64":
        return _loop(medium, nx, ny, nz, 4, "fp64", rng.choice(["x", "y", "z", "xyz"]), pml,
                     cpml=rng.random() < 0.7, state=few and rng.random() < 0.3, **args)
    return _loop(medium, nx, ny, nz, 4, "fp32", dirs, pml, **args)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _dirs(case):
    return ["xyz".index(d) for d in case["dirs"]]


def _steps(case):
    return STRIDE * case["intervals"]


def _problem(case, seed, nx, ny, nz):
    """Solver inputs of one model and the step its run is at."""
    d = 250.0
    deformed = case["kind"] == "deformed"
    pml = {f: case["pml"] for f in ("xmin", "xmax", "ymin", "ymax", "zmax")}
    spec = mesh.MeshSpec(nx=nx, ny=ny, nz=nz, dx=d, dy=d, dz=d, order=case["order"], pml=pml, seed=seed,
                         jitter=0.1 if deformed else 0.0, topo_terms=8 if deformed else 0,
                         topo_amp=0.1 * nz * d if deformed else 0.0)
    if case["kind"] == "halfspace":
        rng = np.random.default_rng(seed)
        vp = float(rng.uniform(4000.0, 6500.0))
        mat = mesh.homogeneous(vp, vp / 1.732, 2700.0)
    else:
        mat = mesh.seeded_layers(seed, nz * d)
        if deformed:
            lo, hi = (-d, -d, -d), (nx * d + d, ny * d + d, nz * d * 1.2 + d)
            mat = mesh.perturbed(mat, mesh.gaussian_field(lo, hi, 0.75 * d, seed + 1), 0.1)
    n = case["tile"]
    tile = ((nx - n) // 2, (ny - n) // 2, n)
    src = np.array([0.46 * nx * d, 0.53 * ny * d, 0.3 * nz * d + 0.1 * d])
    prob = mesh.build_problem(spec, mat, src, nsteps=2000, snapshot_stride=STRIDE, record_depth_max_m=d,
                              record_tile=tile, amp=1.0e13, with_cpml=case["cpml"], device=0,
                              threads=workloads.host_threads())
    # near the peak of the source time function, the last step of a pass a
    # snapshot step
    step = max(0, int(0.9 / prob["dt"]) // STRIDE * STRIDE) + 1
    return prob, step


def _wavefield(prob, d_cell, seed, n_field):
    """Seeded plane waves of 2 to 8 cells' length at the nodes of ``prob``:
    per wavefield u, v, a [node][3]."""
    xyz = np.empty((prob["n_node"], 3))
    xyz[np.asarray(prob["ibool"]).reshape(-1)] = np.asarray(prob["coords"]).reshape(-1, 3)
    x = torch.from_numpy(xyz).cuda()
    rng = np.random.default_rng([seed, 77])
    out = []
    for _ in range(n_field):
        u, v, a = (torch.zeros_like(x) for _ in range(3))
        for _ in range(4):
            k = rng.standard_normal(3)
            k *= 2.0 * math.pi / (d_cell * rng.uniform(2.0, 8.0) * np.linalg.norm(k))
            w = 4000.0 * float(np.linalg.norm(k))
            amp = torch.from_numpy(rng.standard_normal(3)).cuda()
            ph = x @ torch.from_numpy(k).cuda() + float(rng.uniform(0.0, 2.0 * math.pi))
            s, c = torch.sin(ph)[:, None] * amp, torch.cos(ph)[:, None] * amp
            u += s
            v -= w * c
            a -= w * w * s
        out.append(tuple(t.cpu().numpy() for t in (u, v, a)))
    return out


def _sources(case, prob):
    """The source sets of a case: the model's own, then others elsewhere."""
    sets = [{k: prob[k] for k in ("src_cell_ids", "src_weights", "stf")}]
    spec = prob["spec"]
    for q in range(1, case["sources"]):
        at = np.array([(0.3 + 0.15 * q) * spec.nx * spec.dx, 0.4 * spec.ny * spec.dy, (0.25 + 0.1 * q) * spec.nz * spec.dz])
        ids, w = mesh.locate_point_source(prob["coords"], mesh.cell_corners(spec, mesh.vertex_grid(spec)), at,
                                          prob["is_pml"], spec.order)
        stf = mesh.ricker(prob["stf_t"], f0=2.0 + 0.4 * q, t0=1.0, amp=1.0e13)
        sets.append({"src_cell_ids": ids, "src_weights": w, "stf": stf})
    return sets


def _batch_problems(case, seed):
    probs = []
    for k in range(case["models"]):
        n = case["n0"] + 2 * k
        probs.append(_problem(case, seed * 31 + k, n, case["n0"] + 1, max(5, case["n0"] - 2))[0])
    return probs


BATCH_STEP = 51  # step every model of a batch is at


def _elements(case, seed):
    """Random cells by the rules of the element kernel's tests, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nn = (case["order"] + 1) ** 3
    P = case["cells"] * nn

    def uni(*shape):
        return 2.0 * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) - 1.0

    dxi = uni(P, 9) + 3.0 * torch.eye(3, device="cuda", dtype=torch.float64).reshape(1, 9)
    jac = uni(P).abs() + 0.01
    vp, vs, rho = uni(P).abs() + 1000.0, uni(P).abs() + 500.0, uni(P).abs() + 1000.0
    mu = rho * vs * vs
    lam = rho * (vp * vp - 2.0 * vs * vs)
    return {"dxi": dxi, "jac": jac, "lam": lam, "mu": mu, "u": uni(P, 3)}


def prepare(case, seed):
    if case["kind"] == "element":
        lib = gfb.load_library()
        f = lib.gfb_element_residual_noalloc
        f.restype = ctypes.c_int
        f.argtypes = [ctypes.c_int32] + [ctypes.c_void_p] * 4 + [ctypes.c_int32] + [ctypes.c_void_p] * 3
        s = _elements(case, seed)
        s.update(case=case, call=f, r=torch.empty_like(s["u"]))
        return s
    prec = gfb.FP32 if case["precision"] == "fp32" else gfb.FP64
    flags = gfb.FLAG_RECORD_F32 if prec == gfb.FP32 else 0
    dirs = _dirs(case)
    if case["kind"] == "batch":
        probs = _batch_problems(case, seed)
        # finished models leave a batch: none does within these passes
        steps = [10 ** 8 + 100 * k for k in range(len(probs))]
        s = gfb.BatchSolver(probs, dirs=dirs, precision=prec, record_slots=8, flags=flags, n_steps=steps)
        waves = [_wavefield(p, 250.0, seed * 31 + k, len(dirs)) for k, p in enumerate(probs)]
        for f in range(len(dirs)):
            u, v, a = (np.concatenate([waves[k][f][q] for k in s.placement]) for q in range(3))
            s.set_state(f, BATCH_STEP, u, v, a)
    else:
        prob, step = _problem(case, seed, case["nx"], case["ny"], case["nz"])
        if case["sources"] > 1:
            sets = _sources(case, prob)
            n = len(dirs)
            s = gfb.Solver(prob, dirs=dirs * len(sets), precision=prec, record_slots=8, flags=flags, sources=sets,
                           field_source=[f // n for f in range(n * len(sets))])
        else:
            s = gfb.Solver(prob, dirs=dirs, precision=prec, record_slots=8, flags=flags)
        for f, (u, v, a) in enumerate(_wavefield(prob, 250.0, seed, s.n_field)):
            s.set_state(f, step, u, v, a)
    return {"case": case, "solver": s, "dtype": np.float32 if prec == gfb.FP32 else np.float64}


def run(state):
    case = state["case"]
    if case["kind"] == "element":
        st = state["call"](case["cells"], state["dxi"].data_ptr(), state["jac"].data_ptr(), state["lam"].data_ptr(),
                           state["mu"].data_ptr(), case["order"] + 1, state["u"].data_ptr(), state["r"].data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        if st != 0:
            raise RuntimeError(gfb.load_library().gfb_last_error().decode())
        return state["r"]
    s = state["solver"]
    out = {"records": s.run(_steps(case), dtype=state["dtype"])}
    if case["state"]:
        out["state"] = [s.state(f) for f in range(s.n_field)]
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    ng = case["order"] + 1
    nn = ng ** 3
    per_point = 6 * 3 * ng + 60 + 6 * 3 * ng  # gradient, stress and flux, divergence: flops per point and wavefield
    if case["kind"] == "element":
        P = case["cells"] * nn
        return {"bytes": 8.0 * P * (12 + 6), "flops": float(P * per_point)}
    if case["kind"] == "batch":
        boxes = [(case["n0"] + 2 * k, case["n0"] + 1, max(5, case["n0"] - 2)) for k in range(case["models"])]
    else:
        boxes = [(case["nx"], case["ny"], case["nz"])]
    real = 4 if case["precision"] == "fp32" else 8
    F = len(case["dirs"]) * case["sources"]
    o, p = case["order"], case["pml"]
    by = fl = 0.0
    for nx, ny, nz in boxes:
        points = nx * ny * nz * nn
        nodes = (o * nx + 1) * (o * ny + 1) * (o * nz + 1)
        # geometry and materials (12 values), node numbers; displacement (64
        # bits) and velocity read and written, mass
        by += points * (12 * real + 4) + nodes * (3 * F * 2 * (8 + real) + real)
        if case["cpml"]:
            inner = (o * (nx - 2 * p) + 1) * (o * (ny - 2 * p) + 1) * (o * (nz - p) + 1)
            # coefficients of one axis (5 + 3), its memory read and written
            by += (nodes - inner) * real * (8 + 3 * F * 2)
        fl += points * F * per_point + nodes * F * 3 * 8
    rec = case["tile"] ** 2 * nn * F * 15 * real * len(boxes)
    n = _steps(case)
    total = by * n + rec * case["intervals"]
    if case["state"]:
        total += sum((o * nx + 1) * (o * ny + 1) * (o * nz + 1) for nx, ny, nz in boxes) * 9 * F * 8
    return {"bytes": float(total), "flops": float(fl * n)}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------


def _gll(ng):
    """GLL points, weights and D[i, j] = l_j'(x_i), by Newton on P'_N."""
    P = np.polynomial.legendre.Legendre.basis(ng - 1)
    dP, ddP = P.deriv(), P.deriv(2)
    x = -np.cos(math.pi * np.arange(ng) / (ng - 1))
    for _ in range(50):
        x[1:-1] -= dP(x[1:-1]) / ddP(x[1:-1])
    w = 2.0 / (ng * (ng - 1) * P(x) ** 2)
    D = np.zeros((ng, ng))
    for i in range(ng):
        for j in range(ng):
            if i != j:
                D[i, j] = P(x[i]) / (P(x[j]) * (x[i] - x[j]))
    D[0, 0], D[-1, -1] = -ng * (ng - 1) / 4.0, ng * (ng - 1) / 4.0
    return w, D


def _gradient(u, D, dxi):
    """du_c/dx_a [cell, i, j, k, c, a] of u [cell, i, j, k, c]."""
    g = torch.stack([torch.einsum("is,esjkc->eijkc", D, u), torch.einsum("js,eiskc->eijkc", D, u),
                     torch.einsum("ks,eijsc->eijkc", D, u)], -1)
    return torch.einsum("eijkcb,eijkab->eijkca", g, dxi)


def _force(u, D, dxi, jw, lam, mu):
    """-K_e u."""
    G = _gradient(u, D, dxi)
    eye = torch.eye(3, dtype=u.dtype, device=u.device)
    on = (mu > 0.0).to(u.dtype)
    tr = torch.diagonal(G, dim1=-2, dim2=-1).sum(-1)
    sig = ((lam * tr)[..., None, None] * eye + mu[..., None, None] * (G + G.transpose(-1, -2))) * on[..., None, None]
    fl = torch.einsum("eijkca,eijkab->eijkcb", sig, dxi) * jw[..., None, None]
    return -(torch.einsum("si,esjkc->eijkc", D, fl[..., 0]) + torch.einsum("sj,eiskc->eijkc", D, fl[..., 1])
             + torch.einsum("sk,eijsc->eijkc", D, fl[..., 2]))


def _exact_run(prob, cpml, field, waves, step, n_steps, want_state):
    """One wavefield's snapshots and final state from its restart state."""
    ng, nc, nn_ = int(prob["ngll"]), int(prob["n_cell"]), int(prob["n_node"])
    nn = ng ** 3

    def dev(a, *shape):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda().reshape(*shape)

    wq, Dn = _gll(ng)
    D, w3 = dev(Dn, ng, ng), dev(np.einsum("i,j,k->ijk", wq, wq, wq), 1, ng, ng, ng)
    box = (nc, ng, ng, ng)
    dxi = dev(prob["dxi_dx"], *box, 3, 3)
    jw = dev(prob["jacobian"], *box) * w3
    lam, mu = dev(prob["lambda"], *box), dev(prob["mu"], *box)
    ib = torch.from_numpy(np.asarray(prob["ibool"]).reshape(-1).astype(np.int64)).cuda()
    mass = torch.zeros(nn_, dtype=torch.float64, device="cuda").index_add_(0, ib, dev(prob["mass"], -1))
    dt = float(prob["dt"])
    u, v, a = (dev(x, -1, 3) for x in waves)
    damp = None
    if not cpml:
        node = np.zeros(nn_)
        node[np.asarray(prob["ibool"]).reshape(-1)] = np.asarray(prob["damping"]).reshape(-1)
        damp = dev(node, -1, 1)
    else:
        pc = torch.from_numpy(np.nonzero(np.asarray(prob["pml_region"]) != 0)[0]).cuda()
        pib = ib.reshape(nc, nn)[pc].reshape(-1)
        al = dev(prob["pml_coef_alpha"], nc, nn, 3, 3)[pc].reshape(-1, 1, 3, 3)
        A = dev(prob["pml_coef_abar"], nc, nn, 5)[pc].reshape(-1, 1, 5)
        sc = (jw / dev(prob["density"], *box)).reshape(nc, nn)[pc].reshape(-1, 1)
        mem = torch.zeros(pib.numel(), 3, 3, dtype=torch.float64, device="cuda")
        old = torch.zeros(pib.numel(), 3, dtype=torch.float64, device="cuda")
        th = 1.0 / 8.0
        c1, c2 = (1.0 - 2.0 * th) * 0.5 * dt, (1.0 - th) * 0.5 * dt * dt
    rc = torch.from_numpy(np.asarray(prob["recording"]["rec_cell_local"]).astype(np.int64)).cuda()
    rib = ib.reshape(nc, nn)[rc]
    src = field["source"]
    snaps = {"steps": [], "strain": [], "u": [], "v": [], "a": []}
    chunk = 16384
    for t in range(step, step + n_steps):
        ut = u + dt * v + 0.5 * dt * dt * a
        f = torch.zeros_like(u)
        for c0 in range(0, nc, chunk):
            s = slice(c0, min(nc, c0 + chunk))
            ids = ib[c0 * nn : s.stop * nn]
            f.index_add_(0, ids, _force(ut[ids].reshape(-1, ng, ng, ng, 3), D, dxi[s], jw[s], lam[s], mu[s]).reshape(-1, 3))
        if cpml:
            new = u[pib] + c1 * v[pib]
            prev = old + c2 * a[pib]
            f.index_add_(0, pib, sc * (A[..., 0] * v[pib] + A[..., 1] * u[pib] + (A[..., 2:] * mem).sum(-1)))
            mem = al[..., 0] * mem + al[..., 1] * new[..., None] + al[..., 2] * prev[..., None]
            old = new
        else:
            v = torch.where(damp > 0.0, v - damp * v, v)
        if t < len(src["stf"]):
            for cid, w in zip(src["src_cell_ids"], np.asarray(src["src_weights"]).reshape(-1, nn)):
                f[:, field["dir"]].index_add_(0, ib[int(cid) * nn : (int(cid) + 1) * nn], float(src["stf"][t]) * dev(w, -1))
        an = f / mass[:, None]
        u = u + dt * v + 0.5 * dt * dt * a
        v = v + 0.5 * dt * (a + an)
        a = an
        if t % STRIDE == 0:
            G = _gradient(u[rib].reshape(-1, ng, ng, ng, 3), D, dxi[rc]).reshape(len(rc), nn, 3, 3)
            e = 0.5 * (G + G.transpose(-1, -2))
            snaps["steps"].append(t)
            snaps["strain"].append(torch.stack([e[..., 0, 0], e[..., 1, 1], e[..., 2, 2], e[..., 0, 1], e[..., 0, 2], e[..., 1, 2]], -1))
            for k, x in (("u", u), ("v", v), ("a", a)):
                snaps[k].append(x[rib])
    rec = {k: (np.asarray(x, dtype=np.int64) if k == "steps" else torch.stack(x)) for k, x in snaps.items()}
    return rec, (tuple(x.cpu().numpy() for x in (u, v, a)) if want_state else None)


def exact(case, seed):
    if case["kind"] == "element":
        s = _elements(case, seed)
        ng = case["order"] + 1
        w, D = _gll(ng)
        box = (case["cells"], ng, ng, ng)
        w3 = torch.from_numpy(np.einsum("i,j,k->ijk", w, w, w)).cuda()
        r = _force(s["u"].reshape(*box, 3), torch.from_numpy(D).cuda(), s["dxi"].reshape(*box, 3, 3),
                   s["jac"].reshape(box) * w3, s["lam"].reshape(box), s["mu"].reshape(box))
        return r.reshape(-1, 3)
    dirs = _dirs(case)
    if case["kind"] == "batch":
        probs = _batch_problems(case, seed)
        fields = {f: [] for f in range(len(dirs))}
        # snapshots come model after model in the batch's placement order
        for k in reversed(range(len(probs))):
            p = probs[k]
            waves = _wavefield(p, 250.0, seed * 31 + k, len(dirs))
            for f, d in enumerate(dirs):
                fields[f].append(_exact_run(p, True, {"dir": d, "source": p}, waves[f], BATCH_STEP, _steps(case), False)[0])
        rec = {f: {k: (x[0][k] if k == "steps" else torch.cat([m[k] for m in x], 1)) for k in x[0]} for f, x in fields.items()}
        return {"records": rec}
    prob, step = _problem(case, seed, case["nx"], case["ny"], case["nz"])
    sets = _sources(case, prob)
    n = len(dirs)
    waves = _wavefield(prob, 250.0, seed, n * len(sets))
    got = [_exact_run(prob, case["cpml"], {"dir": dirs[f % n], "source": sets[f // n]}, waves[f], step, _steps(case), case["state"])
           for f in range(n * len(sets))]
    out = {"records": {f: r for f, (r, _) in enumerate(got)}}
    if case["state"]:
        out["state"] = [s for _, s in got]
    return out

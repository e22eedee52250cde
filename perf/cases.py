"""The workloads whose speed this framework is judged by, through its public entry points.

A case is a dict of plain values.  Its "kind" is the way a program calls the
library:

* evaluate  one matvec on a plan kept over a fixed geometry (torch tensors on
            the device), with or without the gradient, one or many charge
            vectors, FP64 or FP32 outputs;
* autograd  forward and backward of FMMOperator (charge and position gradients);
* moving    set_geometry + evaluate on new points: a simulation's step, the
            trees and work lists rebuilt every time (plan kept);
* dropin    the reference's fmm(): reference semantics, host arrays, set_geometry
            + evaluate on a plan kept per configuration;
* gmres     the batched BEM solve on a forest of spheres;
* helm      complex Helmholtz or Yukawa matvec (or its transpose).

Point sets: "cube" uniform in [0,1]^3, "clusters" 32 Gaussian clusters of
sigma 0.02 in it, "sphere" uniform on the unit sphere, "ico" the 3-point
quadrature of an icosphere, "forest" centroids of geodesic unit spheres.
"""
import functools
import math

import numpy as np
import torch

import old_fmm_bem_b200 as ob
from old_fmm_bem_b200 import geometry
from old_fmm_bem_b200.autograd import FMMOperator

KERNELS = {"G": ob.LAPLACE_G, "Gni": ob.LAPLACE_GNI, "Gnj": ob.LAPLACE_GNJ, "helmholtz": ob.HELMHOLTZ_G,
           "yukawa": ob.YUKAWA}
SPHERE_BOX = (-1.0001, -1.0001, -1.0001, 2.0002)
UNIT_BOX = (0.0, 0.0, 0.0, 1.0)


def _case(name, kind, kernel, points, n, lmax, p, precision, **more):
    c = dict(name=name, kind=kind, kernel=kernel, points=points, n=n, lmax=lmax, p=p, precision=precision, nrhs=1,
             grad=False, f64=True)
    c.update(more)
    return c


def listed():
    return [
        # the smallest system a program runs (a small molecule's charges): launches and latency
        _case("g_2k_mixed", "evaluate", "G", "cube", 2000, 2, 8, "mixed", grad=True, f64=False),
        # potential and field of a uniform cloud in FP64, the classic FMM test problem
        _case("g_32k_fp64", "evaluate", "G", "cube", 32768, 3, 8, "fp64", grad=True),
        # FP64 with a high order on clustered points: accuracy runs
        _case("g_262k_clusters_fp64", "evaluate", "G", "clusters", 262144, 5, 12, "fp64", grad=True),
        # the headline: forward and backward on a million clustered points
        _case("g_1m_autograd", "autograd", "G", "clusters", 1 << 20, 6, 12, "mixed"),
        # a boundary-element double-layer matvec (the inside of every solver iteration)
        _case("gnj_246k_bem", "evaluate", "Gnj", "ico", 245760, 5, 10, "mixed"),
        # single layer's normal derivative at a surface from charges off it, differentiated: unequal ragged sets
        _case("gni_ragged_autograd", "autograd", "Gni", "mixed_sets", 20011, 4, 10, "mixed", n_src=50021),
        # several charge vectors on one geometry (block methods), odd size
        _case("g_100k_rhs4", "evaluate", "G", "cube", 100003, 3, 10, "mixed", grad=True, nrhs=4),
        # the batched boundary-element solve: 16 molecules-like surfaces, 8 right-hand sides
        _case("gni_forest_gmres", "gmres", "Gni", "forest", 0, 3, 10, "mixed", nrhs=8, nprob=16, tmin=2000,
              tmax=100000, iters=10),
        # a million-point acoustic surface, high order
        _case("helm_1m_mixed", "helm", "helmholtz", "sphere", 1 << 20, 5, 16, "mixed", wavenumber=5.0),
        # a small acoustic problem in full precision, odd size
        _case("helm_30k_fp64", "helm", "helmholtz", "sphere", 30011, 3, 10, "fp64", wavenumber=5.0),
        # the reference program's own call: fmm() on host arrays
        _case("fmm_100k_dropin", "dropin", "G", "cube", 100000, 4, 8, "fp64", grad=True, f64=False),
        # a step of a simulation: the points move, so trees and lists are rebuilt each time
        _case("g_131k_moving", "moving", "G", "clusters", 131071, 5, 10, "mixed", grad=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _depth(points, n, helm=False):
    """The octree depth the library's autotuner arrives at, near enough, for n points of these sets."""
    if points in ("ico", "sphere"):
        d = math.log(n / (900.0 if helm else 240.0)) / math.log(4.0)
    elif points == "clusters":
        d = math.log(n / 4.0) / math.log(8.0)
    else:
        d = math.log(n / 50.0) / math.log(8.0)
    return max(2, min(6, int(round(d))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "autograd", "moving", "dropin", "gmres", "helm", "helm"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "evaluate":
        points = rng.choice(["cube", "clusters", "sphere"])
        kernel = rng.choice(["G", "G", "Gni", "Gnj"])
        n = _log_int(rng, 2000, 1000000 if precision == "mixed" else 200000)
        nrhs = rng.choice([1, 1, 2, 4, 7, 8]) if n < 100000 else 1
        return _case("", kind, kernel, points, n, _depth(points, n), rng.choice([8, 9, 10, 11, 12]), precision,
                     grad=kernel == "G" or (nrhs == 1 and rng.random() < 0.3), nrhs=nrhs, f64=rng.random() < 0.5)
    if kind == "autograd":
        kernel = rng.choice(["G", "Gni", "Gnj"])
        p = rng.choice([8, 10, 12])
        if kernel == "G":
            n = _log_int(rng, 5000, 500000)
            return _case("", kind, "G", "clusters", n, _depth("clusters", n), p, "mixed")
        n, m = _log_int(rng, 5000, 100000), _log_int(rng, 5000, 100000)
        return _case("", kind, kernel, "mixed_sets", n, _depth("clusters", max(n, m)), p, "mixed", n_src=m)
    if kind == "moving":
        points = rng.choice(["cube", "clusters"])
        n = _log_int(rng, 5000, 500000)
        return _case("", kind, "G", points, n, _depth(points, n), rng.choice([8, 10, 12]), "mixed", grad=True)
    if kind == "dropin":
        n = _log_int(rng, 2000, 200000)
        return _case("", kind, rng.choice(["G", "Gni", "Gnj"]), "cube", n, _depth("cube", n), rng.choice([8, 10]),
                     "fp64", f64=False)
    if kind == "gmres":
        return _case("", kind, rng.choice(["Gni", "Gnj"]), "forest", 0, 3, rng.choice([8, 10]), "mixed",
                     nrhs=rng.choice([1, 4, 8]), nprob=rng.choice([1, 5, 12]), tmin=2000,
                     tmax=_log_int(rng, 20000, 100000), iters=rng.choice([5, 10]))
    kernel = rng.choice(["helmholtz", "helmholtz", "yukawa"])
    n = _log_int(rng, 3000, 400000 if precision == "mixed" else 60000)
    return _case("", "helm", kernel, "sphere", n, _depth("sphere", n, True), rng.choice([8, 10, 13, 16]), precision,
                 wavenumber=rng.choice([1.0, 5.0, 9.0]), transpose=rng.random() < 0.3, f64=rng.random() < 0.7)


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=2)
def _ico():
    v, f = geometry.icosphere(6)
    return geometry.quadrature_points(v, f)


@functools.lru_cache(maxsize=4)
def _forest(nprob, tmin, tmax):
    """nprob geodesic spheres, triangle counts log-spaced in [tmin, tmax]: offsets, points, normals, areas."""
    off, xs, ns, ws = [0], [], [], []
    for b in range(nprob):
        t = tmin * (tmax / tmin) ** (b / max(1, nprob - 1))
        v, f = geometry.geodesic_sphere(max(1, int(round((t / 20.0) ** 0.5))))
        x, n, w, _ = geometry.quadrature_points(v, f, "centroid")
        off.append(off[-1] + x.shape[1])
        xs.append(x)
        ns.append(n)
        ws.append(w)
    return np.array(off, np.int32), np.concatenate(xs, 1), np.concatenate(ns, 1), np.concatenate(ws)


def _rotation(rng):
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    return q * np.sign(np.diag(r))


def _unit(rng, n):
    v = rng.standard_normal((3, n))
    return (v / np.linalg.norm(v, axis=0)).astype(np.float32)


def _clusters(rng, n):
    c = rng.uniform(0.1, 0.9, (3, 32))
    lab = rng.integers(0, 32, n)
    return np.clip(c[:, lab] + 0.02 * rng.standard_normal((3, n)), 0.0, 1.0).astype(np.float32)


def _inputs(case, seed):
    """Host inputs: targets, sources, normals of each (or None), root cube, charges, offsets, weights."""
    rng = np.random.default_rng(seed)
    pts, n = case["points"], case["n"]
    box, tn, off, w = UNIT_BOX, None, None, None
    if pts == "cube":
        x = rng.random((3, n), dtype=np.float32)
    elif pts == "clusters":
        x = _clusters(rng, n)
    elif pts == "sphere":
        x, box = _unit(rng, n), SPHERE_BOX
        tn = x.copy()
    elif pts == "ico":
        R = _rotation(rng)
        x0, n0, w, _ = _ico()
        x, tn, box = (R @ x0).astype(np.float32), (R @ n0).astype(np.float32), SPHERE_BOX
    elif pts == "forest":
        R = _rotation(rng)
        off, x0, n0, w = _forest(case["nprob"], case["tmin"], case["tmax"])
        x, tn, box = (R @ x0).astype(np.float32), (R @ n0).astype(np.float32), SPHERE_BOX
    else:  # "mixed_sets": targets on a sphere inside the unit cube, sources in clusters around them
        tn = _unit(rng, n)
        x = (0.5 + 0.35 * tn).astype(np.float32)
    if tn is None:
        tn = _unit(rng, x.shape[1])
    if pts == "mixed_sets":
        xs = _clusters(rng, case["n_src"])
        sn = _unit(rng, case["n_src"])
    else:
        xs, sn = x, tn
    m = xs.shape[1] * case["nrhs"]
    if case["kernel"] == "helmholtz":
        q = (rng.uniform(-1, 1, m) + 1j * rng.uniform(-1, 1, m)).astype(np.complex64)
    elif pts == "ico":  # density per panel x quadrature weight
        q = (np.repeat(rng.uniform(-1, 1, xs.shape[1] // 3), 3) * w).astype(np.float32)
    else:
        q = rng.standard_normal(m).astype(np.float32)
    wt = rng.standard_normal(x.shape[1]).astype(np.float32)  # dL/dpot of the backward passes
    return dict(x=x, xs=xs, tn=tn, sn=sn, same=xs is x, box=box, q=q, wt=wt, off=off, area=w,
                b=rng.uniform(-1, 1, m) if case["kind"] == "gmres" else None)


def _plan(case, semantics=ob.SEM_ACCURATE):
    return ob.Plan(kernel=KERNELS[case["kernel"]], p=case["p"], lmax=case["lmax"],
                   precision=ob.MIXED if case["precision"] == "mixed" else ob.FP64, semantics=semantics,
                   exclude_self=semantics == ob.SEM_ACCURATE, nrhs=case["nrhs"],
                   wavenumber=case.get("wavenumber", 0.0))


def _normals(case, tn, sn):
    return tn if case["kernel"] == "Gni" else None, sn if case["kernel"] == "Gnj" else None


def prepare(case, seed):
    h = _inputs(case, seed)
    st = dict(case=case, box=h["box"], area=h["area"], off=h["off"])
    if case["kind"] == "dropin":  # the reference's caller holds host arrays
        st.update(x=h["x"], tn=h["tn"], q=h["q"], plan=_plan(case, ob.SEM_REFERENCE))
        return st
    dev = {k: torch.from_numpy(h[k]).cuda() for k in ("x", "tn", "sn", "q", "wt")}
    dev["xs"] = dev["x"] if h["same"] else torch.from_numpy(h["xs"]).cuda()
    if h["same"]:
        dev["sn"] = dev["tn"]
    st.update(dev)
    ni, nr = h["x"].shape[1], case["nrhs"]
    tn, sn = _normals(case, dev["tn"], dev["sn"])
    dt = torch.float64 if case["f64"] else torch.float32
    if case["kind"] == "autograd":
        st["q"].requires_grad_(True)
        st["x"].requires_grad_(True)
        st["xs"].requires_grad_(True)
        st["op"] = FMMOperator(st["x"], st["xs"], kernel=KERNELS[case["kernel"]], n_t=tn, n_s=sn, p=case["p"],
                               lmax=case["lmax"], precision=ob.MIXED, bbox=h["box"])
        return st
    st["plan"] = plan = _plan(case)
    if case["kind"] == "gmres":
        plan.set_geometry_batch(h["off"], dev["x"], h["off"], dev["xs"], tn, sn, bbox=h["box"])
        st["weight"] = torch.from_numpy((h["area"] / geometry.E1).astype(np.float32)).cuda()
        st["b"] = torch.from_numpy(h["b"]).cuda()
        return st
    if case["kind"] == "helm":
        cdt = torch.complex128 if case["f64"] else torch.complex64
        st["pot"] = torch.zeros(ni * nr, dtype=cdt if case["kernel"] == "helmholtz" else dt, device="cuda")
    else:
        st["pot"] = torch.zeros(ni * nr, dtype=dt, device="cuda")
        st["grad"] = torch.zeros(3 * ni * nr, dtype=dt, device="cuda") if case["grad"] else None
    if case["kind"] != "moving":
        plan.set_geometry(dev["x"], dev["xs"], tn, sn, bbox=h["box"])
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "evaluate":
        pot, grad = state["plan"].evaluate(state["q"], state["pot"], state["grad"], f64=case["f64"])
        return (pot,) if grad is None else (pot, grad)
    if kind == "autograd":
        q, x, xs = state["q"], state["x"], state["xs"]
        pot = state["op"](q)
        wrt = (q, x) if xs is x else (q, x, xs)
        return (pot.detach(),) + torch.autograd.grad(pot, wrt, state["wt"])
    if kind == "moving":
        state["plan"].set_geometry(state["x"], state["xs"], bbox=state["box"])
        return state["plan"].evaluate(state["q"], state["pot"], state["grad"], f64=case["f64"])
    if kind == "dropin":
        tn, sn = _normals(case, state["tn"], state["tn"])
        state["plan"].set_geometry(state["x"], state["x"], tn, sn, bbox=state["box"])
        pot, grad = state["plan"].evaluate(state["q"])
        return (pot,) if grad is None else (pot, grad)
    if kind == "gmres":  # the residual norms, a diagnostic at rounding level by then, are not compared
        x = torch.zeros_like(state["b"])
        x, iters, _ = state["plan"].gmres(state["b"], x, state["weight"], diag=geometry.BEM_DIAG,
                                          precond=1.0 / geometry.BEM_DIAG, restart=30, max_iter=case["iters"])
        return x, iters
    fn = state["plan"].evaluate_transpose if case.get("transpose") else state["plan"].evaluate
    return fn(state["q"], state["pot"], f64=case["f64"])[0]


# ---------------------------------------------------------------- work
def _grid(x, box, lev):
    g = np.clip(((x.astype(np.float64) - np.array(box[:3])[:, None]) / box[3] * (1 << lev)).astype(np.int64), 0,
                (1 << lev) - 1)
    return np.bincount((g[0] * (1 << lev) + g[1]) * (1 << lev) + g[2], minlength=8 ** lev).reshape((1 << lev,) * 3)


def _nbr(a):
    """Sum over the 27 neighbours of every cell."""
    for ax in range(3):
        pad = [(0, 0)] * 3
        pad[ax] = (1, 1)
        b = np.pad(a, pad)
        n = a.shape[ax]
        a = sum(np.take(b, range(o, o + n), axis=ax) for o in range(3))
    return a


def work(case):
    """Near field: the pairs of neighbouring leaves at 20 flops (a complex pair 30, 8 more per further charge
    vector).  Far field: per box pair of the interaction lists a rotation, an axial translation and a rotation back
    (the least any of the usual translations takes), and twice (p+1)^2 terms per point and component."""
    h = _inputs(case, 0)
    p, nr, lmax = case["p"], case["nrhs"], case["lmax"]
    cplx = case["kind"] == "helm"
    K = (p + 1) ** 2
    rot = sum((2 * n + 1) ** 2 for n in range(p + 1))
    ax = sum((p + 1 - abs(m)) ** 2 for m in range(-p, p + 1))
    per_m2l = 2 * (2 * rot + ax) * (4 if cplx else 1)
    near = far = 0.0
    offs = h["off"] if h["off"] is not None else np.array([0, h["x"].shape[1]])
    for b in range(len(offs) - 1):
        xt = h["x"][:, offs[b]:offs[b + 1]]
        xs = xt if h["same"] else h["xs"]
        near += float((_grid(xt, h["box"], lmax) * _nbr(_grid(xs, h["box"], lmax))).sum())
        for lev in range(2, lmax + 1):
            t, s = (_grid(v, h["box"], lev) > 0 for v in (xt, xs))
            par = _nbr(s.reshape((1 << (lev - 1), 2) * 3).sum(axis=(1, 3, 5)))  # children of the parent's neighbours
            for ax3 in range(3):
                par = par.repeat(2, axis=ax3)
            far += float((t * (par - _nbr(s.astype(np.int64)))).sum())
    ni, nj = h["x"].shape[1], h["xs"].shape[1]
    per_pair = (30.0 if cplx else 20.0) + 8.0 * (nr - 1)
    ncomp = 4 if case["grad"] or case["kind"] == "autograd" else 1
    flops = near * per_pair + nr * (far * per_m2l + 2.0 * K * (nj + ncomp * ni) * (4 if cplx else 1))
    comp = 2 if case["kernel"] == "helmholtz" else 1
    out = 8 if case["f64"] else 4
    nbytes = 12.0 * (ni + nj) + 12.0 * ni * (case["kernel"] in ("Gni", "Gnj"))
    nbytes += nr * comp * (4.0 * nj + out * ncomp * ni)
    if case["kind"] == "autograd":
        flops *= 2
        nbytes += 4.0 * ni + 4.0 * (nj + 3 * nj)
    if case["kind"] == "gmres":
        flops *= case["iters"] + 1
        nbytes += nr * ni * 16.0
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- tolerance
def tolerance(case):
    """About four times what two correct computations at the case's precision were seen to differ by.  Mixed form:
    the FP64 form on the same tree differs by 1e-7 to 4e-7 (FP32 pairs and sums, 22-bit operators), by 1.7e-6 for the
    normal-derivative kernels on surfaces (terms that cancel).  FP64 form: the same points with their axes permuted
    (other operators, the same truncation) differ by 3.2e-15, by 3.7e-14 for the Helmholtz family, whose operators are
    projections.  FP32 outputs add their own rounding.  The solve's operator is near the identity, so its solution
    differs by 1e-8."""
    if case["kind"] == "gmres":
        return {"rel": 1e-7}
    if case["precision"] == "mixed":
        if case["kernel"] in ("Gni", "Gnj") and case["points"] in ("ico", "sphere"):
            return {"rel": 7e-6}
        return {"rel": 1e-6 if case["kind"] == "helm" else 2e-6}
    if not case["f64"]:
        return {"rel": 1e-7}
    return {"rel": 2e-13 if case["kind"] == "helm" else 2e-14}


# ---------------------------------------------------------------- exact
def _direct(kernel, xt, nt, xs, ns, q, k=0.0, ref=False, grad=False):
    """Direct sum in FP64 torch: q (R, nj) -> pot (R, ni), gradients (R, 3, ni) when asked for.  Coincident points
    contribute nothing, except in reference semantics (differences in float, 1e-6f added to r^2, the float pi)."""
    R, ni, nj = q.shape[0], xt.shape[1], xs.shape[1]
    step = max(1, (1 << 26) // nj)
    dt = q.dtype
    pot = torch.empty(R, ni, dtype=dt, device="cuda")
    g = torch.empty(R, 3, ni, dtype=dt, device="cuda") if grad else None
    coef = 0.25 / float(np.float32(math.pi)) if ref else 0.25 / math.pi
    eps = float(np.float32(1e-6)) if ref else 0.0
    for a in range(0, ni, step):
        e = min(ni, a + step)
        if ref:
            d = [(xt[c, a:e, None] - xs[c][None]).double() for c in range(3)]
        else:
            d = [xt[c, a:e, None].double() - xs[c].double()[None] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps
        ri = torch.where(r2 > 0, r2, torch.inf).rsqrt()
        if kernel in ("helmholtz", "yukawa"):
            r = torch.where(r2 > 0, r2, 1.0).sqrt()
            if kernel == "yukawa":  # (pi / 2) e^{-k r} / (k r)
                kv = torch.exp(-k * r) * ri * (0.5 * math.pi / k)
            else:
                kv = torch.polar(ri, k * r) * coef
            pot[:, a:e] = q @ kv.T
            continue
        if kernel == "G":
            pot[:, a:e] = coef * (q @ ri.T)
            if grad:
                r3 = ri * ri * ri
                for c in range(3):
                    g[:, c, a:e] = -coef * (q @ (d[c] * r3).T)
            continue
        n = [v[:, None].double() for v in nt[:, a:e]] if kernel == "Gni" else [v[None].double() for v in ns]
        r3 = ri * ri * ri
        dot = d[0] * n[0] + d[1] * n[1] + d[2] * n[2]
        pot[:, a:e] = coef * (q @ (dot * r3).T)
        if grad:
            c5 = -3.0 * dot * r3 * ri * ri
            for c in range(3):
                g[:, c, a:e] = coef * (q @ (n[c] * r3 + c5 * d[c]).T)
    return pot, g


def _gmres(matvec, b, diag, iters):
    """x minimising the residual of (diag + A) x = b, both sides over diag, over `iters` Krylov steps, per column."""
    V = [b / b.norm(dim=1, keepdim=True)]
    H = torch.zeros(b.shape[0], iters + 1, iters, dtype=torch.float64)
    for j in range(iters):
        w = V[j] + matvec(V[j]) / diag
        for _ in range(2):
            for i in range(j + 1):
                c = (V[i] * w).sum(1)
                H[:, i, j] += c.cpu()
                w = w - c[:, None] * V[i]
        nw = w.norm(dim=1)
        H[:, j + 1, j] = nw.cpu()
        V.append(w / nw[:, None])
    rhs = torch.zeros(b.shape[0], iters + 1, 1, dtype=torch.float64)
    rhs[:, 0, 0] = b.norm(dim=1).cpu()
    y = torch.linalg.lstsq(H, rhs).solution[:, :, 0].cuda()
    return sum(y[:, j:j + 1] * V[j] for j in range(iters))


def exact(case, seed):
    h = _inputs(case, seed)
    if h["x"].shape[1] * float(h["xs"].shape[1]) > 8e10:
        return None  # a quadratic sum of over about 20 seconds
    dev = {k: torch.from_numpy(h[k]).cuda() for k in ("x", "tn", "xs", "sn", "q", "wt")}
    ker, nr, kind = case["kernel"], case["nrhs"], case["kind"]
    x, xs, tn, sn = dev["x"], dev["xs"], dev["tn"], dev["sn"]
    q = dev["q"].reshape(nr, -1).to(torch.complex128 if ker == "helmholtz" else torch.float64)
    if kind == "gmres":
        w = torch.from_numpy((h["area"] / geometry.E1).astype(np.float32)).cuda().double()
        b = torch.from_numpy(h["b"]).cuda().reshape(nr, -1)
        out = torch.empty_like(b)
        for k in range(len(h["off"]) - 1):
            s = slice(int(h["off"][k]), int(h["off"][k + 1]))

            def mv(v, s=s):
                return _direct(ker, x[:, s], tn[:, s], xs[:, s], sn[:, s], (v * w[None, s]).float().double())[0]
            out[:, s] = _gmres(mv, b[:, s] / geometry.BEM_DIAG, geometry.BEM_DIAG, case["iters"])
        return out.reshape(-1), case["iters"]
    if kind == "helm":  # symmetric: the transpose on one point set is the matvec
        pot, _ = _direct(ker, x, None, xs, None, q, k=case["wavenumber"])
        return pot.reshape(-1)
    if kind == "autograd":
        wt = dev["wt"][None].double()
        pot, g = _direct(ker, x, tn, xs, sn, q, grad=True)
        back = {"G": "G", "Gni": "Gnj", "Gnj": "Gni"}[ker]
        sign = 1.0 if ker == "G" else -1.0
        dq, gs = _direct(back, xs, sn, x, tn, wt, grad=True)
        dxt, dxs = wt[0] * g[0], sign * q[0] * gs[0]
        dq = sign * dq[0]
        return (pot[0], dq, dxt + dxs) if h["same"] else (pot[0], dq, dxt, dxs)
    ref = kind == "dropin"
    want = case["grad"] or (ref and ker == "G")
    pot, g = _direct(ker, x, tn, xs, sn, q, ref=ref, grad=want)
    res = (pot.reshape(-1),) if g is None else (pot.reshape(-1), g.reshape(-1))
    return tuple(t.cpu().numpy() for t in res) if ref else res

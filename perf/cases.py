"""The work a user has this library do, as timed cases.

Each case is one call (or one short sequence of calls) through the public
Python API, over the sizes, shapes, kernels and options of the repository's
own workloads and tests:

* ``project``   MLoD projection of device queries (Fastapss.project_device)
* ``host``      projectCPU on host arrays: upload, project, download
* ``protocol``  the application's query-buffer protocol: upload once, then one
                iteration per call, then read the positions back
* ``knn``, ``global``  the other projection modes
* ``build``     a cloud that has just arrived: octree build, kernel, projection
* ``dc``        the dual-contouring field of a resident cell grid
* ``mesh``      the whole dual-contouring pipeline into device vertex buffers
* ``batch``     many resident clouds in one call

Clouds and queries are made on the GPU from the seed.  ``exact`` restates the
projections in float64 with plain torch (its own octree included).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mlodsurfaces_b200 import APSSOctree, DCGrid, Fastapss, FastapssBatch, GlobalAPSS, Kernel

DEV = "cuda"


def listed():
    return [
        # the smallest interactive call: a coarse cloud and one screen patch of
        # queries, where launches and latency count
        _c("project_small", "project", shape="torus", points=10_000, queries=1_000, kernel="gauss", sigma=0.02,
           cutoff=3.0, rule=0, iters=10, depth=12, qpw=1),
        # a host caller projecting a handful of points (projectCPU inside an
        # application's loop): copies, launches and the synchronisation
        _c("host_small", "host", shape="torus", points=20_000, queries=257, kernel="multi4", sigma=0.01, cutoff=3.0,
           rule=1, iters=10, depth=12, qpw=1),
        # the viewer's loop: queries stay on the device, one iteration a frame
        _c("protocol_50k", "protocol", shape="blobs", points=60_000, queries=50_021, kernel="gauss", sigma=0.02,
           cutoff=2.0, rule=0, iters=10, depth=12, qpw=1),
        # the 100k-point torus with the CPU path's semantics; the points are the
        # queries; two queries per warp is what the schedule tuner picks for it
        _c("torus_100k", "project", shape="torus", points=100_000, queries=100_000, kernel="gauss", sigma=0.02,
           cutoff=3.0, rule=1, iters=10, depth=8, qpw=2, on_points=True),
        # an ordinary job at the defaults: rational kernel, default cutoff and
        # schedule, ragged sizes
        _c("rational_500k", "project", shape="knot", points=300_007, queries=500_009, kernel="rational", sigma=1e-3,
           cutoff=2.0, rule=0, iters=5, depth=12, qpw=1),
        # the precision workload: 2M points and queries, four Gaussians, far
        # from the origin, tuned schedule
        _c("precision_2m", "project", shape="blobs", points=2_000_000, queries=2_000_000, kernel="multi4", sigma=0.01,
           cutoff=3.0, rule=0, iters=10, depth=12, qpw=2, far=1000.0),
        # classic APSS over the 32 nearest neighbours
        _c("knn_300k", "knn", shape="blobs", points=300_000, queries=300_000, kernel="multi4", sigma=0.01, k=32,
           iters=10, depth=12),
        # every point weighs in every query
        _c("global_40k", "global", shape="blobs", points=40_000, queries=40_000, kernel="multi4", sigma=0.01, iters=5,
           depth=12),
        # a new cloud: build its octree, project onto it
        _c("build_1m", "build", shape="knot", points=1_000_000, queries=200_003, kernel="multi3", sigma=0.01,
           cutoff=2.0, rule=0, iters=3, depth=12, qpw=1),
        # the signed field of a new scan on a resident depth-8 dual-contouring
        # grid: one projection a corner and a vertex per cell
        _c("dc_field", "dc", shape="knot", points=1_000_000, kernel="rational", sigma=1e-3, cutoff=2.0, rule=0,
           depth=12, grid=8, qpw=2),
        # cloud to mesh: grid generation, field, extraction, two refinements,
        # the result copied into the caller's device buffers (a viewer's)
        _c("mesh_300k", "mesh", shape="knot", points=300_000, kernel="rational", sigma=1e-3, cutoff=2.0, rule=0,
           depth=12, grid=7, qpw=2, rounds=2),
        # 24 resident clouds of mixed sizes and kernels in one call
        _c("batch_24", "batch", clouds=24, small=4_000, large=160_000, iters=10, cutoff=3.0, rule=0, qpw=2),
    ]


def _c(name, kind, **kw):
    return dict(name=name, kind=kind, **kw)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    """A case of the same ranges: sizes log-uniform between the smallest and
    the largest of its kind."""
    kind = rng.choice(["project"] * 6 + ["host", "protocol", "knn", "global", "build", "dc", "mesh", "batch"])
    kernel = rng.choice(["gauss", "multi4", "multi3", "multi8", "rational"])
    sigma = {"gauss": rng.uniform(0.01, 0.03), "rational": 10 ** rng.uniform(-3.3, -2.7)}.get(
        kernel, rng.uniform(0.005, 0.015))
    base = dict(kind=kind, shape=rng.choice(["torus", "blobs", "knot"]), kernel=kernel, sigma=sigma,
                cutoff=rng.choice([2.0, 2.5, 3.0]), rule=rng.choice([0, 0, 1]), iters=rng.choice([1, 3, 5, 10]),
                depth=rng.choice([8, 10, 12, 12]), qpw=rng.choice([1, 1, 2, 2]))
    if kind == "project":
        n = _log(rng, 10_000, 1_200_000)
        base.update(points=n, queries=min(2_000_000, max(1_000, int(n * math.exp(rng.uniform(-2.3, 0.9))))))
        base["depth"] = 12 if n > 300_000 else base["depth"]
    elif kind == "host":
        base.update(points=_log(rng, 10_000, 200_000), queries=_log(rng, 1, 20_000), rule=1)
    elif kind == "protocol":
        n = _log(rng, 10_000, 300_000)
        base.update(points=n, queries=max(1_000, int(n * rng.uniform(0.2, 1.5))))
    elif kind == "knn":
        n = _log(rng, 10_000, 300_000)
        base.update(points=n, queries=max(1_000, int(n * rng.uniform(0.2, 1.0))), k=rng.choice([8, 20, 20, 32]))
    elif kind == "global":
        base.update(points=_log(rng, 5_000, 40_000), queries=_log(rng, 2_000, 40_000), iters=rng.choice([1, 3, 5]))
    elif kind == "build":
        n = _log(rng, 20_000, 1_000_000)
        base.update(points=n, queries=max(1_000, n // 5), iters=rng.choice([1, 3]), depth=12)
    elif kind in ("dc", "mesh"):
        base.update(points=_log(rng, 100_000, 1_000_000 if kind == "dc" else 300_000), kernel="rational",
                    sigma=10 ** rng.uniform(-3.3, -2.7), rule=0, depth=12, cutoff=2.0, shape="knot")
        base["grid"] = rng.choice([6, 7, 8] if kind == "dc" else [5, 6, 7])
        base["rounds"] = rng.choice([1, 2])
    else:
        base = dict(kind="batch", clouds=rng.choice([5, 12, 24, 31]), small=_log(rng, 1_000, 8_000),
                    large=_log(rng, 40_000, 160_000), iters=rng.choice([3, 10]), cutoff=rng.choice([2.0, 3.0]),
                    rule=0, qpw=rng.choice([1, 2]))
    return base


# ---- clouds ------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * (int(seed) % 1_000_000) + 17)
    return g


def _u(g, *s):
    return torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)


def _n(g, *s):
    return torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)


def _cloud(shape, n, g):
    """n points and unit normals (float32) of a noisy surface."""
    if shape == "torus":  # R = 1, r = 0.35, uniform in area, noise 0.002
        m = 2 * n + 256
        u, v, a = _u(g, m) * 2 * math.pi, _u(g, m) * 2 * math.pi, _u(g, m)
        keep = torch.nonzero(a < (1 + 0.35 * torch.cos(v)) / 1.35).flatten()[:n]
        u, v = u[keep], v[keep]
        nv = torch.stack([torch.cos(v) * torch.cos(u), torch.cos(v) * torch.sin(u), torch.sin(v)], 1)
        p = torch.stack([torch.cos(u), torch.sin(u), torch.zeros_like(u)], 1) + 0.35 * nv + 0.002 * _n(g, n, 3)
    elif shape == "knot":  # tube of radius 0.15 around the (2, 3) torus knot, noise 0.002
        m = int(2.2 * n) + 256
        t, th, a = _u(g, m) * 2 * math.pi, _u(g, m) * 2 * math.pi, _u(g, m)

        def tangent(t):
            r = 1 + 0.5 * torch.cos(3 * t)
            dr = -1.5 * torch.sin(3 * t)
            return torch.stack([dr * torch.cos(2 * t) - 2 * r * torch.sin(2 * t),
                                dr * torch.sin(2 * t) + 2 * r * torch.cos(2 * t), 1.5 * torch.cos(3 * t)], 1)

        T = tangent(t)
        sp = T.norm(dim=1)
        keep = torch.nonzero(a < sp / 3.6).flatten()[:n]
        t, th, T = t[keep], th[keep], T[keep] / sp[keep, None]
        N = torch.linalg.cross(T, torch.tensor([0.0, 0.0, 1.0], device=DEV, dtype=torch.float64).expand_as(T))
        N = N / N.norm(dim=1, keepdim=True)
        nv = torch.cos(th)[:, None] * N + torch.sin(th)[:, None] * torch.linalg.cross(T, N)
        r = 1 + 0.5 * torch.cos(3 * t)
        p = torch.stack([r * torch.cos(2 * t), r * torch.sin(2 * t), 0.5 * torch.sin(3 * t)], 1) + 0.15 * nv
        p = p + 0.002 * _n(g, len(p), 3)
    else:  # level set of 12 Gaussian blobs, noise 0.003
        c, rho = _u(g, 12, 3) * 2 - 1, _u(g, 12) * 0.3 + 0.2
        m = n + n // 2 + 256
        j = (_u(g, m) * 12).long()
        d = _n(g, m, 3)
        x = c[j] + (rho[j] * math.sqrt(math.log(2.0)))[:, None] * d / d.norm(dim=1, keepdim=True)

        def field(x):
            f, gr = torch.zeros(len(x), device=DEV, dtype=torch.float64), torch.zeros_like(x)
            for k in range(12):
                dk = x - c[k]
                e = torch.exp(-(dk * dk).sum(1) / rho[k] ** 2)
                f += e
                gr += (-2 / rho[k] ** 2 * e)[:, None] * dk
            return f, gr

        for _ in range(12):
            f, gr = field(x)
            x = x - ((f - 0.5) / (gr * gr).sum(1).clamp_min(1e-9))[:, None] * gr
        f, gr = field(x)
        ok = torch.nonzero(((f - 0.5).abs() < 1e-9) & (gr.norm(dim=1) > 1e-3) & (x.abs().amax(1) < 4)).flatten()
        ok = ok[torch.arange(n, device=DEV) % len(ok)]
        nv = -gr[ok] / gr[ok].norm(dim=1, keepdim=True)
        p = x[ok] + 0.003 * _n(g, n, 3)
    return p, nv.float()


def _inputs(case, seed):
    """Points, normals, queries (float32, GPU) and the points' box diagonal."""
    g = _gen(seed)
    p, nv = _cloud(case["shape"], case["points"], g)
    if case["kind"] in ("dc", "mesh"):  # the application scales a cloud into [-1, 1]^3 first
        p = p - p.mean(0)
        p = p / (p.abs().max() * 1.01)
    diag = float((p.amax(0) - p.amin(0)).norm())
    n = case.get("queries", 0)
    at = torch.arange(n, device=DEV) % case["points"]
    if n > case["points"] or n < case["points"] // 2:
        at = (_u(g, n) * case["points"]).long().clamp_max(case["points"] - 1)
    q = p.float().double()[at] if case.get("on_points") else p[at] + 0.01 * diag * _n(g, n, 3)
    shift = case.get("far", 0.0) * diag / math.sqrt(3.0)
    return (p + shift).float().contiguous(), nv.contiguous(), (q + shift).float().contiguous(), diag


def _kernel(kind, sigma, diag):
    k = Kernel()
    if kind == "gauss":
        k.type, k.sigma = Kernel.GAUSSIAN, sigma * diag
    elif kind == "rational":
        k.type, k.exponent, k.constant_shift = Kernel.SINGULAR, 4.0, sigma
    else:
        k.type = Kernel.GAUSSIAN_MULTIPLE
        k.sigmas = [sigma * diag * 2.0**i for i in range(int(kind[5:]))]
    return k


def _projector(case, tree, kernel, cls=Fastapss):
    f = cls(tree, kernel)
    f.setScalingProtectionSphere(case.get("cutoff", 2.0))
    f.blend_rule = case.get("rule", 0)
    f.queries_per_warp = case.get("qpw", 1)
    return f


# ---- the cases ---------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    p, nv, q, diag = _inputs(case, seed)
    kernel = _kernel(case["kernel"], case["sigma"], diag)
    st = {"case": case, "kernel": kernel, "q": q}
    if kind == "build":
        st.update(p=p, n=nv, out=(torch.empty_like(q), torch.empty_like(q)))
        return st
    tree = APSSOctree()
    if kind == "host":
        tree.build(p.cpu().numpy(), nv.cpu().numpy(), maxDepth=case["depth"])
    else:
        tree.build_device(p, nv, maxDepth=case["depth"])
    if kind == "knn":
        tree.knnMode(True, case["k"])
    st["f"] = f = _projector(case, tree, kernel, GlobalAPSS if kind == "global" else Fastapss)
    if kind in ("host", "protocol"):
        st["q"] = q.cpu().numpy()
        st["out"] = (np.empty_like(st["q"]), np.empty_like(st["q"]))
    elif kind == "dc":
        # the resident grid comes from an earlier scan of the same object
        old = _inputs(case, 0)[0]
        st["grid"] = grid = DCGrid(old, case["grid"])
        st["cells"] = torch.from_numpy(grid.cells).to(DEV)
    elif kind == "mesh":
        cap = 3 * 4 ** (case["grid"] + case["rounds"])
        st["out"] = (torch.zeros(cap, 3, device=DEV), torch.zeros(cap, 3, device=DEV),
                     torch.zeros(2 * cap, 3, dtype=torch.int32, device=DEV))
    else:
        st["out"] = (torch.empty_like(q), torch.empty_like(q))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "host":
        return st["f"].projectCPU(st["q"], case["iters"])
    if kind == "protocol":
        f, n = st["f"], len(st["q"])
        f.copyPointsToGPU(n, st["q"])
        for _ in range(case["iters"] - 1):
            f.project(n, None, None, 1)
        f.project(n, st["out"][0], st["out"][1], 1)
        return st["out"]
    if kind == "build":
        tree = APSSOctree()
        tree.build_device(st["p"], st["n"], maxDepth=case["depth"])
        f = _projector(case, tree, st["kernel"])
        f.project_device(st["q"], st["out"][0], st["out"][1], case["iters"])
        return st["out"][0], st["out"][1], tree.nbOfNodes()
    if kind == "dc":
        cf, vx, nc, nu = st["f"].dc_evaluate_device(st["cells"], st["grid"].max_depth, st["grid"].xform)
        return cf, vx, nc, nu
    if kind == "mesh":
        grid = DCGrid.adaptive(st["f"], case["grid"])
        parts = st["f"].dc_mesh(grid, refine_rounds=case["rounds"]).device_arrays()
        for buf, part in zip(st["out"], parts):
            buf[:len(part)].copy_(part)
        return (*st["out"], len(parts[0]), len(parts[2]))
    if kind == "batch":
        st["b"].project_device(st["counts"], st["q"], st["out"][0], st["out"][1], case["iters"], use_graph=True)
        return st["out"]
    st["f"].project_device(st["q"], st["out"][0], st["out"][1], case["iters"])
    return st["out"]


def _batch_clouds(case, seed):
    """Per-cloud sub-cases: sizes spread over [small, large], shapes, kernels
    and tree depths in turn."""
    out = []
    m = case["clouds"]
    for i in range(m):
        n = int(case["small"] * (case["large"] / case["small"]) ** (i / max(m - 1, 1))) | 1
        kernel = ("gauss", "multi4", "rational", "multi3")[i % 4]
        sigma = {"gauss": 0.02, "rational": 1e-3}.get(kernel, 0.01)
        out.append(dict(kind="project", shape=("torus", "blobs")[i % 2], points=n, queries=n, kernel=kernel,
                        sigma=sigma, cutoff=case["cutoff"], rule=case["rule"], iters=case["iters"],
                        depth=(7, 8, 9, 10, 12)[i % 5], qpw=case["qpw"]))
    return out


def _prepare_batch(case, seed):
    fs, qs = [], []
    for i, c in enumerate(_batch_clouds(case, seed)):
        p, nv, q, diag = _inputs(c, seed * 64 + i)
        tree = APSSOctree()
        tree.build_device(p, nv, maxDepth=c["depth"])
        fs.append(_projector(c, tree, _kernel(c["kernel"], c["sigma"], diag)))
        qs.append(q)
    q = torch.cat(qs).contiguous()
    return {"case": case, "f": fs, "b": FastapssBatch(fs), "q": q, "counts": [len(x) for x in qs],
            "out": (torch.empty_like(q), torch.empty_like(q))}


def work(case):
    """Bytes: inputs once, results once.  Flops: the pair sums where every
    pair is evaluated; for the tree walks about 60 flops per node a query
    visits, and about 1000 such nodes per query and iteration."""
    kind = case["kind"]
    if kind == "batch":
        parts = [work(c) for c in _batch_clouds(case, 0)]
        return {"bytes": sum(w["bytes"] for w in parts), "flops": sum(w["flops"] for w in parts)}
    n, m, it = case["points"], case.get("queries", 0), case.get("iters", 1)
    if kind in ("dc", "mesh"):
        cells = 4 ** case["grid"] * 6
        up = 4 ** case.get("rounds", 0) if kind == "mesh" else 1
        return {"bytes": 64 * n + 60 * cells * up, "flops": 60.0 * 430 * cells * up}
    per = {"knn": 32 * 40.0, "global": 50.0 * n}.get(kind, 60.0 * 1000)
    return {"bytes": 64 * n + 36 * m, "flops": per * m * it}


# ---- float64 restatement ------------------------------------------------------


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mesh", "batch"):
        return None
    p, nv, q, diag = _inputs(case, seed)
    kernel = _kernel(case["kernel"], case["sigma"], diag)
    if kind == "dc":
        return None  # the field's sign pattern decides the other outputs
    if kind == "knn":
        if case["queries"] * case["points"] * case["iters"] > 3e10:
            return None
        return _apss(p, nv, q, kernel, case["iters"], case["k"])
    if kind == "global":
        return _apss(p, nv, q, kernel, case["iters"], 0)
    if case["queries"] * case["iters"] > 3_000_000:
        return None
    tree = _Tree(p, nv, case["depth"])
    x, n = tree.project(q, kernel, case["cutoff"], case["rule"], case["iters"], kind == "protocol")
    return (x, n, tree.n_nodes) if kind == "build" else (x, n)


def _weight(kernel, d2, shift_if_zero=False):
    if kernel.type == Kernel.GAUSSIAN:
        return torch.exp(-d2 / (2.0 * float(np.float32(kernel.sigma)) ** 2)) + kernel.constant_shift
    if kernel.type == Kernel.SINGULAR:
        s = float(np.float32(kernel.constant_shift))
        return max(s, 1e-4) ** kernel.exponent / (d2 + s) ** kernel.exponent
    w = torch.zeros_like(d2)
    for s in kernel.sigmas:
        s = float(np.float32(s))
        w += torch.exp(-d2 / (2.0 * s * s)) / s**3
    return w


def _fit(S, step_max, gpu_rule):
    """Algebraic sphere of the sums in the query frame: the step and normal."""
    Sw, Sn, Sp, Spn, Spp = S[:, 0:1], S[:, 1:4], S[:, 4:7], S[:, 7:8], S[:, 8:9]
    u4 = 0.5 * (Spn - (Sp * Sn).sum(1, True) / Sw) / (Spp - (Sp * Sp).sum(1, True) / Sw)
    u = (Sn - 2 * u4 * Sp) / Sw
    u0 = -((Sp * u).sum(1, True) + u4 * Spp) / Sw
    flat = u4.abs() < (1e-6 if gpu_rule else 1e-12)
    xf = -u * u0 / (u * u).sum(1, True)
    c = u / (-2 * u4)
    rad = ((c * c).sum(1, True) - u0 / u4).clamp_min(0).sqrt()
    xs = c - rad * c / c.norm(dim=1, keepdim=True)
    x = torch.where(flat, xf, xs)
    n = torch.where(flat, Sn, u + 2 * u4 * xs)
    n = n / n.norm(dim=1, keepdim=True)
    ln = x.norm(dim=1, keepdim=True)
    return torch.where(ln > step_max, x * (step_max / ln), x), n


def _apss(p, nv, q, kernel, iters, k):
    """APSS over the k nearest points (k = 0: over all points, weighted by
    their sample areas), float iterates as the path keeps them."""
    P, N = p.double(), nv.double()
    step_max = float((p.amax(0) - p.amin(0)).norm()) / 2
    area = None if k else _Tree(p, nv, 12).area
    x, nrm = q.double(), torch.zeros_like(q, dtype=torch.float64)
    chunk = max(1, int(2.0e8 / len(P)))
    for it in range(iters):
        xs, ns = [], []
        for s in range(0, len(q), chunk):
            y = x[s:s + chunk].float().double() if k else x[s:s + chunk]
            if k:
                d2 = sum((P[:, a] - y[:, a:a + 1]) ** 2 for a in range(3))
                d2, i = d2.topk(min(k, len(P)), dim=1, largest=False)
                d = P[i] - y[:, None]
                S = _sums(_weight(kernel, d2), N[i], d, d2)
            else:
                d2 = sum((P[:, a] - y[:, a:a + 1]) ** 2 for a in range(3))
                w = _weight(kernel, d2) * area
                W = w.sum(1, True)
                wp, wn = w @ P, w @ N
                pn, pp = (P * N).sum(1), (P * P).sum(1)
                Sp = wp - W * y
                Spn = (w @ pn)[:, None] - (wn * y).sum(1, True)
                Spp = (w * d2).sum(1, True)
                S = torch.cat([W, wn, Sp, Spn, Spp], 1)
            st, n = _fit(S, step_max, False)
            xs.append(y + st)
            ns.append(n)
        x, nrm = torch.cat(xs), torch.cat(ns)
    return x, nrm


def _sums(w, n, d, d2):
    return torch.cat([w.sum(1, True), (w[..., None] * n).sum(1), (w[..., None] * d).sum(1),
                      (w * (d * n).sum(2)).sum(1, True), (w * d2).sum(1, True)], 1)


class _Tree:
    """The octree in float64: the tight box halved per axis (bounds and splits
    are floats), one point per leaf or the depth limit, moments per node."""

    def __init__(self, p, nv, D):
        lo, hi = p.amin(0).cpu().numpy(), p.amax(0).cpu().numpy()
        cells, bounds = [], []
        for a in range(3):
            b = np.array([lo[a], hi[a]], np.float32)
            levels, x = [b], p[:, a].double()
            k = torch.zeros(len(p), dtype=torch.long, device=DEV)
            for _ in range(D):
                s = (b[:-1] + b[1:]).astype(np.float32).astype(np.float64) / 2.0
                k = 2 * k + (x > torch.from_numpy(s).to(DEV)[k]).long()
                nb = np.empty(2 * len(b) - 1, np.float32)
                nb[0::2], nb[1::2] = b, s.astype(np.float32)
                b = nb
                levels.append(b)
            cells.append(k)
            bounds.append([torch.from_numpy(v.astype(np.float64)).to(DEV) for v in levels])
        self.origin = torch.from_numpy((lo.astype(np.float64) + hi) / 2).to(DEV)
        e = (hi - lo).astype(np.float32)
        self.step_max = float(np.linalg.norm(e)) / 2
        P, N = p.double() - self.origin, nv.double()
        n = len(p)
        own = torch.zeros(n, dtype=torch.long, device=DEV)  # each point's node on the level
        alive = torch.ones(n, dtype=torch.bool, device=DEV)
        lev, base = [], 0
        area = torch.zeros(n, dtype=torch.float64, device=DEV)
        leaf_of = torch.zeros(n, dtype=torch.long, device=DEV)
        for d in range(D + 1):
            idx = torch.nonzero(alive).flatten()
            if not len(idx):
                break
            c = [(cells[a][idx] >> (D - d)) for a in range(3)]
            code = torch.zeros(len(idx), dtype=torch.long, device=DEV)
            for b in range(d - 1, -1, -1):
                code = (code << 3) | ((c[0] >> b) & 1) | (((c[1] >> b) & 1) << 1) | (((c[2] >> b) & 1) << 2)
            u, inv, cnt = torch.unique(code, sorted=True, return_inverse=True, return_counts=True)
            first = torch.zeros(len(u), dtype=torch.long, device=DEV)
            first[inv] = torch.arange(len(idx), device=DEV)
            box = [(bounds[a][d][c[a][first]], bounds[a][d][c[a][first] + 1]) for a in range(3)]
            r2 = sum((h - l) ** 2 for l, h in box)
            ctr = torch.stack([(l + h) / 2 - self.origin[a] for a, (l, h) in enumerate(box)], 1)
            parent = own[idx][first]
            leaf = (cnt == 1) | (d == D)
            lev.append(dict(ctr=ctr, r=r2.sqrt() / 2, cnt=cnt, leaf=leaf, parent=parent, base=base))
            own[idx] = base + inv
            pl = leaf[inv]
            area[idx[pl]] = (r2 / cnt)[inv][pl]
            leaf_of[idx[pl]] = (base + inv)[pl]
            alive[idx[pl]] = False
            base += len(u)
        self.n_nodes, self.area = base, area
        cat = lambda key: torch.cat([v[key] for v in lev])  # noqa: E731
        self.ctr, self.r, self.leaf, self.parent = cat("ctr"), cat("r"), cat("leaf"), cat("parent")
        self.cnt = cat("cnt")
        # point records of the leaves that hold several points
        multi = self.leaf & (self.cnt > 1)
        pts = torch.nonzero(multi[leaf_of]).flatten()
        pts = pts[torch.sort(leaf_of[pts], stable=True)[1]]
        # raw moments about the origin, bottom up, then centred
        raw = torch.zeros(base, 9, dtype=torch.float64, device=DEV)
        m = torch.cat([area[:, None], area[:, None] * N, area[:, None] * P, (area * (P * N).sum(1))[:, None],
                       (area * (P * P).sum(1))[:, None]], 1)
        raw.index_add_(0, leaf_of, m)
        for v in reversed(lev[1:]):
            s = slice(v["base"], v["base"] + len(v["cnt"]))
            raw.index_add_(0, v["parent"], raw[s].clone())
        self.raw = torch.cat([raw, m[pts]])
        ex = len(pts)
        self.ctr = torch.cat([self.ctr, P[pts]])
        self.r = torch.cat([self.r, torch.zeros(ex, dtype=torch.float64, device=DEV)])
        self.leaf = torch.cat([self.leaf, torch.ones(ex, dtype=torch.bool, device=DEV)])
        self.multi = torch.cat([multi, torch.zeros(ex, dtype=torch.bool, device=DEV)])
        self.par = torch.cat([self.parent, leaf_of[pts]])
        kids = torch.bincount(self.par[1:], minlength=base + ex)
        self.kids = kids
        order = torch.sort(self.par[1:], stable=True)[1] + 1
        self.child = order
        self.off = torch.cumsum(kids, 0) - kids
        self.bar = self.raw[:, 4:7] / self.raw[:, 0:1]

    def _at(self, nodes, y):
        """Sums of the nodes with every point equally weighted, in the query frame."""
        r = self.raw[nodes]
        Sp = r[:, 4:7] - r[:, 0:1] * y
        Spn = r[:, 7:8] - (r[:, 1:4] * y).sum(1, True)
        Spp = r[:, 8:9] - 2 * (r[:, 4:7] * y).sum(1, True) + r[:, 0:1] * (y * y).sum(1, True)
        return torch.cat([r[:, 0:4], Sp, Spn, Spp], 1)

    def sums(self, y, kernel, cutoff, rule):
        n = len(y)
        S = torch.zeros(n, 9, dtype=torch.float64, device=DEV)
        qi = torch.arange(n, device=DEV)
        node = torch.zeros(n, dtype=torch.long, device=DEV)
        f = torch.ones(n, dtype=torch.float64, device=DEV)
        while len(qi):
            yq = y[qi]
            dist = (self.ctr[node] - yq).norm(dim=1)
            w = _weight(kernel, ((self.bar[node] - yq) ** 2).sum(1))
            cr = cutoff * self.r[node]
            multi = self.multi[node]
            term = (self.leaf[node] & ~multi) | (~self.leaf[node] & (dist > cr))
            S.index_add_(0, qi[term], (f * w)[term, None] * self._at(node[term], yq[term]))
            op = torch.nonzero(~term).flatten()
            if not len(op):
                break
            k = self.kids[node[op]]
            src = torch.repeat_interleave(op, k)
            start = torch.cumsum(k, 0) - k
            j = torch.arange(len(src), device=DEV) - torch.repeat_interleave(start, k)
            ch = self.child[torch.repeat_interleave(self.off[node[op]], k) + j]
            blend = ~multi[src]
            dP = (cr - dist)[src]
            dC = ((self.ctr[ch] - y[qi[src]]).norm(dim=1) - cutoff * self.r[ch]).clamp_min(0)
            t = dP / (dP + dC)
            beta = torch.where(blend, 0.5 - 0.5 * torch.cos(math.pi * t), torch.ones_like(t))
            rho = self.raw[ch, 0] / self.raw[node[src], 0] if rule == 0 else 1.0 / self.kids[node[src]].double()
            K = torch.zeros(len(qi), dtype=torch.float64, device=DEV)
            K.index_add_(0, src, (1 - beta) * rho * (f * w)[src])
            S.index_add_(0, qi[op], K[op, None] * self._at(node[op], yq[op]))
            fc = f[src] * beta
            if rule == 1:  # the CPU rule weighs only the last point of a leaf
                last = j == (self.kids[node[src]] - 1)
                fc = torch.where(multi[src] & ~last, torch.zeros_like(fc), fc)
            qi, node, f = qi[src], ch, fc
        return S

    def project(self, q, kernel, cutoff, rule, iters, world_iterates):
        out, nrm = [], []
        for s in range(0, len(q), 16384):
            y = q[s:s + 16384].double() - self.origin
            n = torch.zeros_like(y)
            for _ in range(iters):
                st, n = _fit(self.sums(y, kernel, cutoff, rule), self.step_max, rule == 0)
                y = y + st
                if world_iterates:  # the query buffer holds floats between calls
                    y = (y + self.origin).float().double() - self.origin
            out.append(y + self.origin)
            nrm.append(n)
        return torch.cat(out), torch.cat(nrm)

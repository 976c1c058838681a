"""The packet walk (calls of many queries, two or more iterations): 32 queries
share a walk and the order is taken anew after the first iteration.  A query's
result may depend on neither, so every way to run the same call gives the same
bits; FP64 gives the values."""
import ctypes as C

import numpy as np
import pytest

import oracle
from conftest import make_kernel, rel_err
from mlodsurfaces_b200 import APSSOctree, Fastapss, FastapssBatch, ProjectionServer, synth
from mlodsurfaces_b200 import _capi as capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL_DIAG = 1e-5  # the projection's parity bar against FP64
N = 350_001      # ragged: the last packet holds one query


def project(f, q, iters):
    d_q = torch.from_numpy(np.ascontiguousarray(q, np.float32)).cuda()
    p, n = torch.full_like(d_q, float("nan")), torch.full_like(d_q, float("nan"))
    f.project_device(d_q, p, n, iters)
    torch.cuda.synchronize()
    return p.cpu().numpy(), n.cpu().numpy()


def equal(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.fixture(scope="module")
def cloud():
    pts, nrm = synth.torus(40000, seed=41)
    pts = synth.make_tie_free(pts)
    t = APSSOctree()
    t.build(pts, nrm)
    q = np.concatenate([synth.perturbed_queries(pts, 0.01, seed=s) for s in range(9)])[:N]
    return pts, nrm, t, q


@pytest.mark.parametrize("kind,rule,qpw,depth,min_depth", [
    ("gauss", 0, 1, 12, 0), ("multi", 0, 1, 12, 3), ("singular", 1, 1, 12, 0), ("multi", 1, 1, 4, 0),
    ("gauss", 0, 2, 12, 0), ("gauss", 1, 4, 5, 0)])
def test_matches_fp64(cloud, kind, rule, qpw, depth, min_depth):
    """Depths 4 and 5: leaves of hundreds of points, walked in chunks of 8."""
    pts, nrm, _, q = cloud
    if qpw > 1:  # shared walks change to packets at 800k queries
        q = np.concatenate([q, q + np.float32(1e-4), q - np.float32(1e-4)])
    diag = synth.bbox_diag(pts)
    k = make_kernel(kind, diag)
    t = APSSOctree()
    t.build(pts, nrm, maxDepth=depth)
    f = Fastapss(t, k)
    f.setScalingProtectionSphere(3.0)
    f.setMinDepth(min_depth)
    f.blend_rule = rule
    f.queries_per_warp = qpw
    p, n = project(f, q, 3)
    st = f.last_stats()
    assert st["iterations"] == 3 * len(q) and st["overflows"] == 0
    assert st["lane_visits"] < st["node_visits"] / 8  # the walk was shared by more than eight queries
    sel = np.random.default_rng(1).choice(len(q), 400, replace=False)
    want, wn = oracle.OracleTree(pts, nrm, depth).project_mlod(q[sel], 3, k, rule=rule, cutoff=3.0, min_depth=min_depth)
    assert rel_err(p[sel], want, diag).max() < TOL_DIAG
    assert ((n[sel] * wn).sum(1) > 1 - 1e-4).all()


@pytest.mark.parametrize("iters", [2, 5])
def test_same_bits_however_it_is_run(cloud, iters):
    pts, _, t, q = cloud
    q = q.copy()
    q[5], q[77] = np.nan, 1e25  # fail in their first iteration and stay where they are
    k = make_kernel("multi", synth.bbox_diag(pts))
    f = Fastapss(t, k)
    want = project(f, q, iters)
    assert np.isnan(want[0][5]).all() and np.array_equal(want[0][77], q[77])
    assert (want[1][[5, 77]] == 0).all() and np.isfinite(want[1]).all()
    perm = np.random.default_rng(2).permutation(N)
    got = project(f, q[perm], iters)
    assert equal([x[np.argsort(perm)] for x in got], want)
    f.reorder = False
    assert equal(project(f, q, iters), want)
    f.reorder = True
    f.converge = capi.CONVERGE_EXACT
    assert equal(project(f, q, iters), want)
    f.converge = capi.CONVERGE_OFF
    f.copyPointsToGPU(N, q)  # in place
    out = np.empty_like(q), np.empty_like(q)
    f.project(N, out[0], out[1], iters)
    assert equal(out, want)
    d_q = torch.from_numpy(q).cuda()
    out = torch.empty_like(d_q), torch.empty_like(d_q)
    capi.check(capi.load().mlods_project_device_noalloc(t.handle, N, capi.ptr(d_q), capi.ptr(out[0]), capi.ptr(out[1]),
                                                        iters, C.c_float(-1.0), C.c_void_p(0)))
    torch.cuda.synchronize()
    assert equal([x.cpu().numpy() for x in out], want)
    small = project(f, q[:3000], iters)
    for graph in (False, True):
        b = FastapssBatch([f, f, f])
        d_q = torch.from_numpy(np.concatenate([q[:3000], q, q[:3000]])).cuda()
        out = torch.empty_like(d_q), torch.empty_like(d_q)
        for _ in range(2):
            b.project_device([3000, N, 3000], d_q, out[0], out[1], iters, use_graph=graph)
        torch.cuda.synchronize()
        got = [x.cpu().numpy() for x in out]
        assert equal([x[3000:3000 + N] for x in got], want)
        assert equal([x[:3000] for x in got], small) and equal([x[3000 + N:] for x in got], small)
        assert b.last_stats()["walk_launches"] == 3
    srv = ProjectionServer([f], n_streams=2, max_batch_queries=90000)  # the request runs in pieces
    try:
        tickets = [srv.submit(0, q, iters), srv.submit(0, q[:3000], iters)]
        assert equal(srv.wait(tickets[0], 60000)[:2], want) and equal(srv.wait(tickets[1], 60000)[:2], small)
    finally:
        srv.close()

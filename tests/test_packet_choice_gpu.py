"""Calls large enough for packets walk in them unless more than an eighth of the
queries lie far from the cloud; every way to run a call decides alike."""
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
N = 350_003


@pytest.fixture(scope="module")
def cloud():
    pts, nrm = synth.torus(40000, seed=91)
    pts = synth.make_tie_free(pts)
    t = APSSOctree()
    t.build(pts, nrm)
    k = make_kernel("multi", synth.bbox_diag(pts))
    f = Fastapss(t, k)
    f.setScalingProtectionSphere(3.0)
    q = np.concatenate([synth.perturbed_queries(pts, 0.01, seed=s) for s in range(9)])[:N]
    return pts, nrm, t, f, k, q


def with_far(pts, q, count):
    """`count` of the queries moved outside the box widened by half its extent."""
    q = q.copy()
    rng = np.random.default_rng(3)
    at = rng.choice(len(q), count, replace=False)
    lo, hi = pts.min(0), pts.max(0)
    ext = (hi - lo).max()
    q[at, rng.integers(0, 3, count)] = (hi.max() + ext * rng.uniform(0.6, 3.0, count)).astype(np.float32)
    return q


def project(f, q, iters):
    d_q = torch.from_numpy(np.ascontiguousarray(q, np.float32)).cuda()
    p, n = torch.full_like(d_q, float("nan")), torch.full_like(d_q, float("nan"))
    f.project_device(d_q, p, n, iters)
    torch.cuda.synchronize()
    return p.cpu().numpy(), n.cpu().numpy()


def equal(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("far,packets", [(0, True), (N // 8, True), (N // 8 + 1, False), (N, False)])
def test_decision(cloud, far, packets):
    pts, nrm, t, f, k, q = cloud
    q = with_far(pts, q, far)
    want = project(f, q, 2)
    st = f.last_stats()
    assert st["overflows"] == 0 and st["iterations"] <= 2 * N
    assert (st["lane_visits"] < 0.5 * st["node_visits"]) == packets
    if not packets:  # the walk of smaller calls, bit for bit
        part = project(f, q[:100_000], 2)
        assert equal(part, [w[:100_000] for w in want])
    sel = np.random.default_rng(1).choice(N, 300, replace=False)
    ref, rn = oracle.OracleTree(pts, nrm, 12).project_mlod(q[sel], 2, k, rule=0, cutoff=3.0)
    ok = np.linalg.norm(rn, axis=1) > 0.5
    near = np.abs(q[sel]).max(1) <= np.abs(pts).max() + 0.1  # far fits amplify rounding
    assert rel_err(want[0][sel][ok & near], ref[ok & near], synth.bbox_diag(pts)).max(initial=0) < TOL_DIAG
    # in place, without an order, without allocation, in a batch, served
    f.reorder = False
    assert equal(project(f, q, 2), want)
    f.reorder = True
    out = np.empty_like(q), np.empty_like(q)
    f.copyPointsToGPU(N, q)
    f.project(N, out[0], out[1], 2)
    assert equal(out, want)
    d_q = torch.from_numpy(q).cuda()
    out = torch.empty_like(d_q), torch.empty_like(d_q)
    capi.check(capi.load().mlods_project_device_noalloc(t.handle, N, capi.ptr(d_q), capi.ptr(out[0]), capi.ptr(out[1]),
                                                        2, C.c_float(-1.0), C.c_void_p(0)))
    torch.cuda.synchronize()
    assert equal([x.cpu().numpy() for x in out], want)
    d_q = torch.from_numpy(np.concatenate([q[:3000], q, q])).cuda()
    out = torch.empty_like(d_q), torch.empty_like(d_q)
    b = FastapssBatch([f, f, f])
    for graph in (False, True):
        b.project_device([3000, N, N], d_q, out[0], out[1], 2, use_graph=graph)
        torch.cuda.synchronize()
        got = [x.cpu().numpy()[3000:] for x in out]
        assert equal([x[:N] for x in got], want) and equal([x[N:] for x in got], want)
    srv = ProjectionServer([f], n_streams=2)
    try:
        assert equal(srv.wait(srv.submit(0, q, 2))[:2], want)
    finally:
        srv.close()


def test_replayed_graph_decides_on_its_inputs(cloud):
    """A captured call holds both walks; which one runs follows the queries."""
    pts, _, _, f, _, q = cloud
    far = with_far(pts, q, N // 2)
    want = project(f, q, 2), project(f, far, 2)
    s = torch.cuda.Stream()
    d_q = torch.from_numpy(q).cuda()
    p, n = torch.empty_like(d_q), torch.empty_like(d_q)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        f.project_device(d_q, p, n, 2, stream=s.cuda_stream)
        s.synchronize()
        with torch.cuda.graph(g, stream=s):
            f.project_device(d_q, p, n, 2, stream=s.cuda_stream)
    for src, w in ((far, want[1]), (q, want[0]), (far, want[1])):
        d_q.copy_(torch.from_numpy(src))
        p.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert equal([p.cpu().numpy(), n.cpu().numpy()], w)

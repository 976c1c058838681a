"""Which form a one-query-per-warp projection walks in -- 64 nodes a round only
where that pays -- and the forms' results where each is at its edge."""
import numpy as np
import pytest

import oracle
from conftest import make_kernel, rel_err
from mlodsurfaces_b200 import APSSOctree, Fastapss, FastapssBatch, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL_DIAG = 1e-5  # the projection's parity bar against FP64


def project(f, q, iters):
    d_q = torch.from_numpy(np.ascontiguousarray(q, np.float32)).cuda()
    p, n = torch.full_like(d_q, float("nan")), torch.full_like(d_q, float("nan"))
    f.project_device(d_q, p, n, iters)
    torch.cuda.synchronize()
    return p.cpu().numpy(), n.cpu().numpy()


def projector(pts, nrm, depth, cutoff, min_depth=0, rule=0, kind="multi", diag=None):
    t = APSSOctree()
    t.build(pts, nrm, maxDepth=depth)
    k = make_kernel(kind, diag or synth.bbox_diag(pts))
    f = Fastapss(t, k)
    f.setScalingProtectionSphere(cutoff)
    f.setMinDepth(min_depth)
    f.blend_rule = rule
    return f, k


@pytest.mark.parametrize("n,depth,cutoff,min_depth,wide", [
    (2000, 12, 3.0, 0, True), (2000, 12, 2.0, 4, True), (40000, 12, 2.5, 0, True), (2000, 12, 6.0, 0, True),
    (16384, 12, 2.0, 0, True), (16385, 12, 2.0, 0, False), (8192, 12, 1.5, 0, True), (8193, 12, 1.5, 0, False),
    (2369, 12, 6.5, 0, False), (2369, 12, 3.0, 5, False), (2369, 3, 3.0, 0, False), (2368, 12, 6.5, 0, True),
    (2368, 12, 9.5, 0, False), (2368, 12, 3.0, 5, True), (2368, 12, 3.0, 6, False)])
def test_form_and_fp64(n, depth, cutoff, min_depth, wide):
    pts, nrm = synth.torus(20000, seed=31)
    pts = synth.make_tie_free(pts)
    q = np.concatenate([synth.perturbed_queries(pts, 0.01, seed=s) for s in (32, 33)])[:n]
    f, k = projector(pts, nrm, depth, cutoff, min_depth)
    p, _ = project(f, q, 1)
    narrow = f.last_stats()["rounds"]  # one iteration: 32 nodes a round
    project(f, p, 1)
    narrow += f.last_stats()["rounds"]
    p, m = project(f, q, 2)
    st = f.last_stats()
    if wide:
        assert st["rounds"] < 0.95 * narrow
    else:  # (but for the world coordinates' rounding in between)
        assert abs(st["rounds"] - narrow) < 0.005 * narrow
    assert st["overflows"] == 0
    sel = np.random.default_rng(1).choice(n, 100, replace=False)
    want, wn = oracle.OracleTree(pts, nrm, depth).project_mlod(q[sel], 2, k, rule=0, cutoff=cutoff, min_depth=min_depth)
    assert rel_err(p[sel], want, synth.bbox_diag(pts)).max() < TOL_DIAG
    assert ((m[sel] * wn).sum(1) > 1 - 1e-4).all()


def test_batch_and_calls_take_the_same_form():
    """On both sides of the line in the number of queries."""
    pts, nrm = synth.torus(20000, seed=41)
    f, _ = projector(synth.make_tie_free(pts), nrm, 12, 2.0)
    q = synth.perturbed_queries(pts, 0.01, seed=42)
    counts = [len(q), 16384, 3000]
    want = [project(f, q[:c], 2) for c in counts]
    d_q = torch.from_numpy(np.concatenate([q[:c] for c in counts])).cuda()
    out = torch.empty_like(d_q), torch.empty_like(d_q)
    FastapssBatch([f, f, f]).project_device(counts, d_q, out[0], out[1], 2)
    torch.cuda.synchronize()
    for j in range(2):
        assert np.array_equal(out[j].cpu().numpy(), np.concatenate([w[j] for w in want]))


@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("points", [31, 32, 33, 63, 64, 65, 97, 400])
def test_leaf_wider_than_a_round(points, rule):
    """A leaf of many points in a tree of small ones, which 64-node rounds walk."""
    pts, nrm = synth.torus(8000, seed=51)
    pts = synth.make_tie_free(pts).astype(np.float32)
    pts = np.concatenate([pts, np.repeat(pts[100:101], points - 1, 0)])
    nrm = np.concatenate([nrm, np.repeat(nrm[100:101], points - 1, 0)])
    q = synth.perturbed_queries(pts[:8000], 0.01, seed=52)[:100]
    q[:50] = pts[100] + 0.02 * (q[:50] - pts[:50])
    f, k = projector(pts, nrm, 12, 3.0, rule=rule)
    p, m = project(f, q, 3)
    st = f.last_stats()
    assert st["overflows"] == 0
    want, wn = oracle.OracleTree(pts, nrm, 12).project_mlod(q, 3, k, rule=rule, cutoff=3.0)
    assert rel_err(p, want, synth.bbox_diag(pts)).max() < TOL_DIAG
    assert ((m * wn).sum(1) > 1 - 1e-4).all()


def test_last_point_alone_of_a_tree_of_one_leaf():
    """The CPU rule weighs a leaf's last point alone, and one sample defines no
    sphere: a query that fails stays where the failing iteration began."""
    pts, nrm = synth.torus(3000, seed=3000)
    pts = synth.make_tie_free(pts)
    f, _ = projector(pts, nrm, 0, 3.0, rule=1)
    q = synth.perturbed_queries(pts, 0.01, seed=6)[:300]
    first = project(f, q, 1)[0]
    p, m = project(f, q, 2)
    assert f.last_stats()["overflows"] == 0 and np.isfinite(p).all()
    failed = np.linalg.norm(m, axis=1) < 0.5
    assert ((p[failed] == q[failed]).all(1) | (p[failed] == first[failed]).all(1)).all()


def test_tuner_times_what_the_schedule_decides():
    """From 800,000 queries on every schedule walks in packets; the pick must
    still be that of the walks without them, where sharing pays."""
    pts, nrm = synth.torus(60000, seed=61)
    f, _ = projector(synth.make_tie_free(pts), nrm, 12, 3.0)
    q = np.concatenate([synth.perturbed_queries(pts, 0.01, seed=s) for s in range(14)])
    d_q = torch.from_numpy(q).cuda()
    res = f.tune_schedule(d_q, 2)
    assert res["queries_per_warp"] > 1 and f.queries_per_warp == res["queries_per_warp"]
    assert res["ms"][1] > 1.15 * min(res["ms"].values())
    before = project(f, q, 2)  # and calls still walk in packets
    st = f.last_stats()
    assert st["lane_visits"] < st["node_visits"] / 8
    f.queries_per_warp = 1
    assert all(np.array_equal(a, b) for a, b in zip(project(f, q, 2), before))

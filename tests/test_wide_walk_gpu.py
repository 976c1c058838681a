"""The wide walk (one query per warp, two nodes a lane; two or more iterations)
where its rounds can go wrong: multi-point leaves wider than a warp, trees of a
few nodes, nodes opened whatever their distance, NaN queries, and the rule that a query's result does not depend on its launch."""
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


@pytest.mark.parametrize("n,depth,min_depth", [(1, 12, 0), (2, 12, 0), (9, 12, 0), (3000, 0, 0), (3000, 1, 0),
                                               (3000, 3, 2), (3000, 12, 5), (40000, 12, 0)])
@pytest.mark.parametrize("rule", [0, 1])
def test_matches_fp64(n, depth, min_depth, rule):
    pts, nrm = synth.torus(max(n, 16), seed=n + depth)
    pts, nrm = synth.make_tie_free(pts)[:n], nrm[:n]
    q = synth.perturbed_queries(synth.torus(300, seed=5)[0], 0.01, seed=6)
    diag = synth.bbox_diag(synth.torus(300, seed=5)[0])
    k = make_kernel("multi", diag)
    t = APSSOctree()
    t.build(pts, nrm, maxDepth=depth)
    f = Fastapss(t, k)
    f.setScalingProtectionSphere(3.0)
    f.setMinDepth(min_depth)
    f.blend_rule = rule
    p, m = project(f, q, 4)
    want, wn = oracle.OracleTree(pts, nrm, depth).project_mlod(q, 4, k, rule=rule, cutoff=3.0, min_depth=min_depth)
    if (rule, depth) == (1, 0):
        return  # the CPU rule weighs one point of a tree of one leaf: no sphere to compare
    ok = np.linalg.norm(wn, axis=1) > 0.5
    assert np.array_equal(np.linalg.norm(m, axis=1) > 0.5, ok)
    if n >= 3000:  # a handful of points fits spheres that amplify rounding
        assert rel_err(p[ok], want[ok], diag).max() < TOL_DIAG
    assert f.last_stats()["overflows"] == 0


def test_nan_query_fails_alone():
    pts, nrm = synth.torus(20000, seed=11)
    q = synth.perturbed_queries(pts, 0.01, seed=12)[:500]
    t = APSSOctree()
    t.build(synth.make_tie_free(pts), nrm)
    f = Fastapss(t, make_kernel("gauss", synth.bbox_diag(pts)))
    want = project(f, q, 3)
    q[7] = np.nan
    p, n = project(f, q, 3)
    keep = np.arange(500) != 7
    assert np.isnan(p[7]).all() and (n[7] == 0).all()
    assert np.array_equal(p[keep], want[0][keep]) and np.array_equal(n[keep], want[1][keep])


@pytest.mark.parametrize("iters", [1, 2, 5])
def test_result_does_not_depend_on_the_launch(iters):
    pts, nrm = synth.torus(20000, seed=21)
    t = APSSOctree()
    t.build(synth.make_tie_free(pts), nrm)
    f = Fastapss(t, make_kernel("multi", synth.bbox_diag(pts)))
    q = synth.perturbed_queries(pts, 0.01, seed=22)[:5000]
    p, n = project(f, q, iters)
    for a, b in ((0, 1), (17, 50), (1000, 5000)):
        pp, nn = project(f, q[a:b], iters)
        assert np.array_equal(pp, p[a:b]) and np.array_equal(nn, n[a:b])
    d_q = torch.from_numpy(q).cuda()
    bp, bn = torch.empty_like(d_q), torch.empty_like(d_q)
    FastapssBatch([f, f]).project_device([1200, 3800], d_q, bp, bn, iters)
    assert np.array_equal(bp.cpu().numpy(), p) and np.array_equal(bn.cpu().numpy(), n)

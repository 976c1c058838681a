"""Which walk a served request takes: its tree's settings and its own size decide,
not the requests that share a batch with it."""
import numpy as np
import pytest

from conftest import make_kernel
from mlodsurfaces_b200 import APSSOctree, Fastapss, ProjectionServer, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def projectors():
    """One and two queries per warp."""
    out = []
    for qpw in (1, 2):
        pts, nrm = synth.torus(30000, seed=70 + qpw)
        t = APSSOctree()
        t.build(synth.make_tie_free(pts), nrm)
        f = Fastapss(t, make_kernel("multi", synth.bbox_diag(pts)))
        f.setScalingProtectionSphere(3.0)
        f.queries_per_warp = qpw
        q = np.concatenate([synth.perturbed_queries(pts, 0.01, seed=s) for s in range(14)])
        out.append((f, q))
    return out


def alone(f, q, iters):
    f.copyPointsToGPU(len(q), q)
    p, n = np.empty_like(q), np.empty_like(q)
    f.project(len(q), p, n, iters)
    return p, n


def test_pieces_do_not_follow_their_batch(projectors):
    """400,000 queries on the first tree in two pieces, the second of which
    shares its batch with requests on the other tree."""
    (f, q), (g, r) = projectors
    q = q[:400_000]
    want = alone(f, q, 3)
    srv = ProjectionServer([f, g], n_streams=1)
    try:
        big = srv.submit(0, q, 3)
        small = [srv.submit(1, r[1000 * i:1000 * (i + 1)], 3) for i in range(8)]
        got = srv.wait(big)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        for t in small:
            srv.wait(t)
        assert srv.stats()["batches"] < 10  # they did share one
    finally:
        srv.close()


def test_small_pieces_do_not_walk_in_packets(projectors):
    """Pieces that leave most of the GPU idle in packets take the walk of a call
    of their own size; all pieces of a request take the same."""
    (f, q), _ = projectors
    q = q[:400_000]
    want = alone(f, q, 2)  # in packets
    small = [alone(f, q[i:i + 5000], 2) for i in range(0, len(q), 5000)]
    small = [np.concatenate([s[j] for s in small]) for j in (0, 1)]
    assert not np.array_equal(small[0], want[0])
    for batch, same in ((1 << 14, small), (79_999, small), (80_000, want), (1 << 18, want)):
        srv = ProjectionServer([f], n_streams=2, max_batch_queries=batch)
        try:
            got = srv.wait(srv.submit(0, q, 2))
            assert np.array_equal(got[0], same[0]) and np.array_equal(got[1], same[1]), batch
        finally:
            srv.close()

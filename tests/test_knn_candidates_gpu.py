"""The neighbour searches' candidate buffer where it fills, empties and spills
over: clouds smaller than a warp, than the neighbour count, leaves of many
points (ranges wider than a warp), and queries far from everything."""
import numpy as np
import pytest

from mlodsurfaces_b200 import APSSOctree, synth
from test_gather_gpu import assert_knn_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth", [(1, 12), (31, 12), (33, 12), (65, 12), (700, 0), (5000, 2), (20000, 4), (20000, 12)])
@pytest.mark.parametrize("k", [1, 7, 31, 32])
def test_sets_match_bruteforce(n, depth, k):
    pts, nrm = synth.torus(max(n, 2), seed=n + depth)
    pts, nrm = synth.make_tie_free(pts)[:n], nrm[:n]
    t = APSSOctree()
    t.build(pts, nrm, maxDepth=depth)
    q = synth.perturbed_queries(synth.torus(120, seed=k)[0], 0.05, seed=k)
    q[:4] = [[9, 9, 9], [-40, 0, 0], [0, 0, 0], [0, 0, 500]]
    assert_knn_sets(pts, q, k, t)

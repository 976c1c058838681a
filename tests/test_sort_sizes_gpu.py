"""The device radix sort at the sizes where its forms change: one block (1, 2,
4 or 8 items a thread), tiles added up by column, tiles scanned.  Key-value
sorts show in the octree's point order (equal codes keep the input order) and
in the query order (every query projected once), key sorts in the cell grid."""
import numpy as np
import pytest

import oracle
from conftest import make_kernel
from mlodsurfaces_b200 import APSSOctree, DCGrid, Fastapss, synth
from mlodsurfaces_b200.apss import _cuda_available

pytestmark = pytest.mark.gpu

SIZES = [1023, 1025, 2048, 2049, 4097, 8192, 8193, 128 * 2048, 128 * 2048 + 1]


@pytest.mark.parametrize("n", SIZES)
def test_point_order(n):
    """Depth 3: at most 512 distinct codes, so the order inside a leaf is the
    sort's stability."""
    pts, nrm = synth.torus(n, seed=n)
    pts = synth.make_tie_free(pts, 3)
    t = APSSOctree()
    t.build(pts, nrm, maxDepth=3)
    dev, ora = t.export(), oracle.OracleTree(pts, nrm, 3).export()
    for k in ("perm", "leaf_off", "leaf_cnt", "first_child"):
        assert np.array_equal(dev[k], ora[k]), k


@pytest.mark.parametrize("n", SIZES)
def test_query_order_is_a_permutation(n):
    pts, nrm = synth.torus(2000, seed=3)
    t = APSSOctree()
    t.build(synth.make_tie_free(pts), nrm)
    q = np.repeat(synth.perturbed_queries(pts, 0.01, seed=n), n // 2000 + 1, axis=0)[:n]
    out = []
    for reorder in (True, False):
        f = Fastapss(t, make_kernel("gauss", synth.bbox_diag(pts)))
        f.reorder = reorder
        f.copyPointsToGPU(n, q)
        p, m = np.full((n, 3), np.nan, np.float32), np.full((n, 3), np.nan, np.float32)
        f.project(n, p, m, 1)
        out.append((p, m))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("depth,span", [(6, 1.0), (9, 1.0), (14, 1.0), (12, 7.0)])
def test_cell_grid(depth, span):
    """Cell keys packed into 32 bits, into more, and sets of one block; points
    outside the unit zone give negative and large coordinates."""
    assert _cuda_available()
    pts, _ = synth.torus(9000, seed=depth)
    pts = (span * synth.normalize_like_pn(pts)).astype(np.float32)
    dev, host = DCGrid(pts, depth, device=True), DCGrid(pts, depth, device=False)
    assert np.array_equal(dev.cells, host.cells)

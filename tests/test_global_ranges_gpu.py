"""The global projection's split over ranges of whole tiles (256 points): last
tiles of one point, one range, one range a tile, more tiles than ranges."""
import numpy as np
import pytest

import oracle
from conftest import TOL_DIAG, make_kernel, rel_err
from mlodsurfaces_b200 import APSSOctree, GlobalAPSS, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,nq", [(255, 40), (512, 300), (513, 300), (769, 1), (5121, 257), (17000, 600), (20480, 300)])
@pytest.mark.parametrize("kind", ["gauss", "multi"])
def test_matches_fp64(n, nq, kind):
    pts, nrm = synth.torus(n, seed=n)
    pts = synth.make_tie_free(pts)
    q = np.resize(synth.perturbed_queries(pts, 0.01, seed=nq), (nq, 3)).astype(np.float32)
    diag = synth.bbox_diag(pts)
    k = make_kernel(kind, diag)
    t = APSSOctree()
    t.build(pts, nrm)
    d_q = torch.from_numpy(q).cuda()
    p, m = torch.empty_like(d_q), torch.empty_like(d_q)
    GlobalAPSS(t, k).project_device(d_q, p, m, 2)
    torch.cuda.synchronize()
    sel = np.arange(nq)[:: max(1, nq // 40)]
    want, _ = oracle.OracleTree(pts, nrm, 12).project_global(q[sel], 2, k)
    assert rel_err(p.cpu().numpy()[sel], want, diag).max() < TOL_DIAG

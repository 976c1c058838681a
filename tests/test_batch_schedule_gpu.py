"""Which trees of a batch get launches of their own: the library's choice until a
schedule is set or tuned, then the schedule's, where 0 means none."""
import numpy as np
import pytest

from conftest import make_kernel
from mlodsurfaces_b200 import APSSOctree, Fastapss, FastapssBatch, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
COUNTS = [40_000, 5_000, 5_000]  # the first fills the GPU's walks four times over


@pytest.fixture(scope="module")
def setup():
    fs, qs = [], []
    for i, n in enumerate(COUNTS):
        pts, nrm = synth.torus(20000, seed=80 + i)
        t = APSSOctree()
        t.build(synth.make_tie_free(pts), nrm)
        f = Fastapss(t, make_kernel(["gauss", "multi", "singular"][i], synth.bbox_diag(pts)))
        f.setScalingProtectionSphere(3.0)
        f.queries_per_warp = 2
        fs.append(f)
        qs.append(np.concatenate([synth.perturbed_queries(pts, 0.01, seed=s) for s in (1, 2)])[:n])
    return fs, qs


def run(b, qs, iters=2):
    d_q = torch.from_numpy(np.concatenate(qs)).cuda()
    out = torch.empty_like(d_q), torch.empty_like(d_q)
    b.project_device(COUNTS, d_q, out[0], out[1], iters)
    torch.cuda.synchronize()
    return out


def test_own_choice_and_none(setup):
    fs, qs = setup
    want = [[], []]
    for f, q in zip(fs, qs):
        d_q = torch.from_numpy(q).cuda()
        out = torch.empty_like(d_q), torch.empty_like(d_q)
        f.project_device(d_q, out[0], out[1], 2)
        for w, o in zip(want, out):
            w.append(o)
    want = [torch.cat(w) for w in want]
    b = FastapssBatch(fs)
    first = b.schedule()
    assert 5_000 < first["solo_min_queries"] <= 40_000
    for solo, launches in ((None, 2), (0, 1), (5_000, 3), (40_001, 1), (first["solo_min_queries"], 2)):
        if solo is not None:
            b.set_schedule(solo_min_queries=solo)
        got = run(b, qs)
        st = b.last_stats()
        assert st["walk_launches"] == launches, solo
        assert st["solo_min_queries"] == (first["solo_min_queries"] if solo is None else solo)
        assert all(torch.equal(g, w) for g, w in zip(got, want))


def test_tuner_tries_the_shared_launch(setup):
    fs, qs = setup
    b = FastapssBatch(fs)
    d_q = torch.from_numpy(np.concatenate(qs)).cuda()
    out = torch.empty_like(d_q), torch.empty_like(d_q)
    b.tune(COUNTS, d_q, out[0], out[1], 2)
    cands = [tuple(v for k, v in c.items() if k != "ms") for c in b.tune_results()]
    assert len(set(cands)) == 7
    for c in b.tune_results():
        b.set_schedule(c["queries_per_warp"], bool(c["reorder"]), c["grid_pct"], c["line_order"] == "by specialisation",
                       c["solo_min_queries"])
        run(b, qs)
        assert b.last_stats()["walk_launches"] == (2 if 0 < c["solo_min_queries"] <= 40_000 else 1)


def test_one_query_forms_are_counted(setup):
    """One query per warp: below a cutoff of 2.5 the tree with many queries walks
    32 nodes at a time and the others 64, in a launch each."""
    fs, qs = setup
    saved = [f.getScalingProtectionSphere() for f in fs]
    try:
        for f in fs:
            f.queries_per_warp = 1
            f.setScalingProtectionSphere(2.0)
        b = FastapssBatch(fs)
        run(b, qs)
        assert b.last_stats()["walk_launches"] == 2 and b.schedule()["solo_min_queries"] == 0
    finally:
        for f, c in zip(fs, saved):
            f.queries_per_warp = 2
            f.setScalingProtectionSphere(c)

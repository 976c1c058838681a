"""Memory of trees, batches and meshes: freeing one leaves the stream captures of
other threads alone, is refused where cudaFree is (and made up for later), mesh
arrays can be shared as cudaMalloc's can, and a device reset ends what is kept."""
import ctypes as C
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import ROOT, make_kernel
from mlodsurfaces_b200 import APSSOctree, DCGrid, Fastapss, synth
from mlodsurfaces_b200 import _capi as capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GLOBAL, THREAD_LOCAL = 0, 1  # cudaStreamCaptureMode
CAPTURE_INVALIDATED = 901    # cudaErrorStreamCaptureInvalidated


def cudart():
    torch.cuda.init()
    return C.CDLL("libcudart.so.12")


class Capture:
    """A capture open on a stream of its own; `result` is what ending it returned."""

    def __init__(self, rt, mode):
        self.rt, self.mode, self.stream = rt, mode, torch.cuda.Stream()

    def __enter__(self):
        assert self.rt.cudaStreamBeginCapture(C.c_void_p(self.stream.cuda_stream), self.mode) == 0
        return self

    def __exit__(self, *exc):
        g = C.c_void_p(0)
        self.result = self.rt.cudaStreamEndCapture(C.c_void_p(self.stream.cuda_stream), C.byref(g))
        if g.value:
            self.rt.cudaGraphDestroy(g)
        self.rt.cudaGetLastError()


def make(n, seed):
    pts, nrm = synth.torus(n, seed=seed)
    t = APSSOctree()
    t.build(synth.make_tie_free(pts), nrm)
    return t, synth.perturbed_queries(pts, 0.01, seed=seed + 1)[:2000], make_kernel("gauss", synth.bbox_diag(pts))


def project(t, q, k):
    return Fastapss(t, k).projectCPU(q, 3)


def in_thread(fn):
    err = []

    def run():
        try:
            fn()
        except BaseException as e:  # noqa: BLE001 -- handed to the caller
            err.append(e)

    th = threading.Thread(target=run)
    th.start()
    th.join(60)
    assert not th.is_alive() and not err, err


def test_free_leaves_another_threads_capture_alone():
    rt = cudart()
    t0, q, k = make(20000, 1)
    want = project(t0, q, k)
    t1 = make(20000, 3)[0]
    got = []

    def work():
        t1.free()
        t2 = make(20000, 1)[0]  # (takes up what was freed)
        got.append(project(t2, q, k))
        t2.free()

    with Capture(rt, THREAD_LOCAL) as c:
        in_thread(work)
    assert c.result == 0
    for r in (got[0], project(t0, q, k)):
        assert all(np.array_equal(a, b) for a, b in zip(r, want))


def test_refused_free_is_made_up_for():
    """A capture in global mode refuses cudaFree (and ends); the block must not
    be handed out without the wait, nor be lost."""
    rt = cudart()
    capi.check(capi.load().mlods_release_scratch())
    t0, q, k = make(200000, 5)
    want = project(t0, q, k)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    t1 = make(200000, 7)[0]
    with Capture(rt, GLOBAL) as c:
        t1.free()
    assert c.result == CAPTURE_INVALIDATED
    for _ in range(2):
        t2 = make(200000, 5)[0]
        assert all(np.array_equal(a, b) for a, b in zip(project(t2, q, k), want))
        t2.free()
    capi.check(capi.load().mlods_release_scratch())
    # (the driver hands memory out in pieces of 2 MiB)
    assert torch.cuda.mem_get_info()[0] >= before - (4 << 20)


def test_mesh_arrays_can_be_shared():
    t, _, k = make(20000, 9)
    f = Fastapss(t, k)
    parts = f.dc_mesh(DCGrid.adaptive(f, 4), refine_rounds=1).device_arrays()
    cu = C.CDLL("libcuda.so.1")
    for part in parts:
        ok = C.c_int(0)  # CU_POINTER_ATTRIBUTE_IS_LEGACY_CUDA_IPC_CAPABLE
        assert cu.cuPointerGetAttribute(C.byref(ok), 10, C.c_uint64(part.data_ptr())) == 0
        assert ok.value == 1


RESET = """
import ctypes as C
import numpy as np
import torch  # noqa: F401 -- brings libcudart
from mlodsurfaces_b200 import APSSOctree, Fastapss, GlobalAPSS, Kernel, synth
pts, nrm = synth.torus(20000, seed=1)
pts = synth.make_tie_free(pts)
q = synth.perturbed_queries(pts, 0.01, seed=2)[:2000]
k = Kernel()
k.type, k.sigma = Kernel.GAUSSIAN, 0.05

def run():
    t = APSSOctree()
    t.build(pts, nrm)
    out = (*Fastapss(t, k).projectCPU(q, 3), *GlobalAPSS(t, k).projectCPU(q, 2))
    t.free()
    return out

before = run()
assert C.CDLL("libcudart.so.12").cudaDeviceReset() == 0
for _ in range(2):
    assert all(np.array_equal(a, b) for a, b in zip(run(), before))
"""


def test_works_on_after_a_device_reset():
    """Kept blocks and the scratch pool end with their context."""
    res = subprocess.run([sys.executable, "-c", RESET], cwd=ROOT, capture_output=True, text=True, timeout=240)
    assert res.returncode == 0, res.stderr


def test_many_small_objects():
    """Kept blocks are found and given up by size and age, not by a walk of all."""
    pts, nrm = synth.torus(64, seed=11)
    pts = synth.make_tie_free(pts)
    torch.cuda.synchronize()
    for _ in range(2):
        trees = []
        for _ in range(300):
            t = APSSOctree()
            t.build(pts, nrm)
            trees.append(t)
        assert len({t.nbOfNodes() for t in trees}) == 1
        for t in trees:
            t.free()
    capi.check(capi.load().mlods_release_scratch())

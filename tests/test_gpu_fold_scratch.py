"""GPU tests of where eb_fold_arrivals takes its scratch from: a pool that the process set
for the device serves it; a device reset leaves it (and the allocation-free form) working;
under stream capture the scratch belongs to the graph, which replays."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.test_gpu_fold import host_fold

pytestmark = pytest.mark.gpu

# A process of its own: both cases change what the whole process uses.
CHILD = r"""
import ctypes, glob, site, sys
import numpy as np
from edlut_b200 import _lib
found = [f for d in site.getsitepackages() for f in glob.glob(d + "/nvidia/cuda_runtime/lib/libcudart.so*")]
rt = ctypes.CDLL(found[0] if found else "/usr/local/cuda/lib64/libcudart.so")
L = _lib.load()

def ok(rc):
    assert rc == 0, rc

rng = np.random.default_rng(2)
n, m = 3000, 70
target, kind = rng.integers(0, m, n).astype(np.int32), rng.integers(0, 3, n).astype(np.int8)
weight, time = rng.random(n).astype(np.float32), rng.integers(0, 9, n) * 1e-5
want = np.zeros((3, m), np.float32)
for i in np.lexsort((np.arange(n), time)):
    want[kind[i], target[i]] += weight[i]

def device(x):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(x.nbytes)))
    ok(rt.cudaMemcpy(p, x.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(x.nbytes), 1))
    return p

def fold(op):
    d = [device(x) for x in (target, kind, weight, time)]
    g = [device(np.zeros(m, np.float32)) for _ in range(3)]
    s = ctypes.c_void_p()
    ok(rt.cudaStreamCreate(ctypes.byref(s)))
    _lib.check(op(s, n, *d, m, *g))
    ok(rt.cudaStreamSynchronize(s))
    out = np.zeros((3, m), np.float32)
    for a, p in zip(out, g):
        ok(rt.cudaMemcpy(a.ctypes.data_as(ctypes.c_void_p), p, ctypes.c_size_t(a.nbytes), 2))
    np.testing.assert_array_equal(out, want)

if sys.argv[1] == "reset":
    for op in (L.eb_fold_arrivals, L.eb_fold_arrivals_noalloc):
        fold(op)
    ok(rt.cudaDeviceReset())
    for op in (L.eb_fold_arrivals, L.eb_fold_arrivals_noalloc, L.eb_fold_arrivals):
        fold(op)
else:
    class Props(ctypes.Structure):  # cudaMemPoolProps
        _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("locType", ctypes.c_int),
                    ("locId", ctypes.c_int), ("security", ctypes.c_void_p), ("rest", ctypes.c_ubyte * 64)]
    fold(L.eb_fold_arrivals)
    props = Props(1, 0, 1, 0)  # pinned memory of device 0
    pool = ctypes.c_void_p()
    ok(rt.cudaMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)))
    ok(rt.cudaDeviceSetMemPool(0, pool))
    fold(L.eb_fold_arrivals)
    high = ctypes.c_uint64()
    ok(rt.cudaMemPoolGetAttribute(pool, 8, ctypes.byref(high)))  # cudaMemPoolAttrUsedMemHigh
    assert high.value >= 16 * n, high.value
print("done")
"""


@pytest.mark.parametrize("case", ["reset", "set_pool"])
def test_scratch_follows_the_device(case):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD, case], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stdout + r.stderr


def test_captured_fold_replays():
    import torch
    from edlut_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng(3)
    n, m = 5000, 300
    target = rng.integers(0, m, n).astype(np.int32)
    target[:40] = 7  # one list beyond what a thread keeps itself
    stype, weight, time = rng.integers(0, 3, n).astype(np.int8), rng.random(n).astype(np.float32), rng.integers(0, 5, n) * 1e-5
    dev = [torch.from_numpy(x).cuda() for x in (target, stype, weight, time)]
    g0 = [rng.random(m).astype(np.float32) for _ in range(3)]
    out = [torch.from_numpy(x.copy()).cuda() for x in g0]
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        _lib.check(L.eb_fold_arrivals(ctypes.c_void_p(s.cuda_stream), n, *(x.data_ptr() for x in dev), m,
                                      *(x.data_ptr() for x in out)))
    want = g0
    for _ in range(3):
        graph.replay()
        want = host_fold(target, stype, weight, time, m, want)
    torch.cuda.synchronize()
    for a, b in zip(out, want):
        np.testing.assert_array_equal(a.cpu().numpy(), b)

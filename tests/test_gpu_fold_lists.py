"""GPU test of the fold's per-target lists: as many arrivals per target as a thread keeps
itself, one fewer and one more, several targets beyond it at once, ties in time and no
times at all, from two streams at a time; bit for bit the host's per-arrival fold."""
import ctypes

import numpy as np
import pytest

from tests.test_gpu_fold import host_fold

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("timed", [True, False])
@pytest.mark.parametrize("counts", [(15,), (16,), (17,), (1, 16, 0, 17, 40, 33, 2)])
def test_lists_of_every_length(counts, timed):
    import torch
    from edlut_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng(len(counts))
    m = len(counts)
    target = rng.permutation(np.repeat(np.arange(m), counts)).astype(np.int32)
    n = len(target)
    stype = rng.integers(0, 3, n).astype(np.int8)
    weight = rng.random(n).astype(np.float32)
    time = rng.integers(0, 4, n) * 1e-5
    g0 = [rng.random(m).astype(np.float32) for _ in range(3)]
    want = host_fold(target, stype, weight, time if timed else np.zeros(n), m, g0)
    dev = [torch.from_numpy(x).cuda() for x in (target, stype, weight, time)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[torch.from_numpy(x.copy()).cuda() for x in g0] for _ in range(2)]
    torch.cuda.synchronize()
    for s, out in zip(streams, outs):
        _lib.check(L.eb_fold_arrivals(ctypes.c_void_p(s.cuda_stream), n, *(x.data_ptr() for x in dev[:3]),
                                      dev[3].data_ptr() if timed else None, m, *(x.data_ptr() for x in out)))
    torch.cuda.synchronize()
    for out in outs:
        for a, b in zip(out, want):
            np.testing.assert_array_equal(a.cpu().numpy(), b)


@pytest.mark.parametrize("timed", [True, False])
@pytest.mark.parametrize("counts", [(95,), (96,), (97,), (3, 96, 97, 0, 16, 129, 1, 17), (1000, 1025) + 40 * (110,), 200 * (2,) + (4097,),
                                    tuple(110 if 64 <= t < 104 else 1 for t in range(18944))])
def test_lists_that_a_warp_sorts(counts, timed):
    """Lists just below, at and beyond what a thread sorts, alone and several in a warp; and
    more of them in one warp (full of targets from 18,944 on) than it takes one by one."""
    import torch
    from edlut_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng([len(counts), sum(counts)])
    m = len(counts)
    target = rng.permutation(np.repeat(np.arange(m), counts)).astype(np.int32)
    n = len(target)
    stype = rng.integers(0, 3, n).astype(np.int8)
    weight = rng.random(n).astype(np.float32)
    time = rng.integers(0, 9, n) * 1e-5
    g0 = [rng.random(m).astype(np.float32) for _ in range(3)]
    want = host_fold(target, stype, weight, time if timed else np.zeros(n), m, g0)
    dev = [torch.from_numpy(x).cuda() for x in (target, stype, weight, time)]
    out = [torch.from_numpy(x.copy()).cuda() for x in g0]
    torch.cuda.synchronize()
    _lib.check(L.eb_fold_arrivals(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), n, *(x.data_ptr() for x in dev[:3]),
                                  dev[3].data_ptr() if timed else None, m, *(x.data_ptr() for x in out)))
    torch.cuda.synchronize()
    for a, b in zip(out, want):
        np.testing.assert_array_equal(a.cpu().numpy(), b)

"""Batches that mix curve codes launch their codes side by side on helper streams
kept in a process-wide pool: contexts in several threads, on the default and on
their own streams, more of them than the pool keeps, against one at a time."""
import concurrent.futures as cf

import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def run(seed, stream=None):
    b = ds.uneven_batch(150, seed=seed, max_ctrl=120, max_samples=200)
    out = []
    for _ in range(3):
        with g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_MIXED, rtol=b.rtol, stream=stream) as calc:
            calc.createArclengthTable()
            pos = torch.from_numpy(b.sample_positions()).cuda()
            cnt = torch.from_numpy(b.n_samples).cuda()
            u = torch.empty_like(pos)
            torch.cuda.synchronize()
            calc.arclengthReverseInto(cnt, pos, u)
            calc.synchronize()
            out.append((calc.getAllCurveArclengths(), u.cpu().numpy()))
    for L, u in out[1:]:
        np.testing.assert_array_equal(L, out[0][0])
        np.testing.assert_array_equal(u, out[0][1])
    return out[0]


@pytest.mark.parametrize("own_stream", [False, True])
def test_contexts_in_threads(own_stream, gpu_lib):
    want = [run(s) for s in range(8)]

    def job(s):
        return run(s, torch.cuda.Stream() if own_stream else None)

    with cf.ThreadPoolExecutor(8) as ex:
        got = list(ex.map(job, range(8)))
    for (L0, u0), (L1, u1) in zip(want, got):
        np.testing.assert_array_equal(L0, L1)
        np.testing.assert_array_equal(u0, u1)


def test_many_contexts_alive(gpu_lib):
    b = ds.uneven_batch(60, seed=3, max_ctrl=60, max_samples=64)
    calcs = [g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_MIXED) for _ in range(9)]
    L = []
    for c in calcs:
        c.createArclengthTable()
    for c in calcs:
        L.append(c.getAllCurveArclengths())
        c.close()
    g.release_cached_memory()
    for x in L[1:]:
        np.testing.assert_array_equal(x, L[0])
    with g.ArclengthCalculateGpu.from_batch(b, precision=g.GCV_MIXED) as c:
        c.createArclengthTable()
        np.testing.assert_array_equal(c.getAllCurveArclengths(), L[0])

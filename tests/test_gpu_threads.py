"""Threads with contexts and streams of their own: tables, samplings and captured steps
that are created and destroyed while other threads capture theirs give the results of
the same calls made alone, bit for bit."""
import threading

import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import datasets as ds
from gcurval_gb300 import learned
from test_gpu_graph_pools import device

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FORMS = [dict(precision=g.GCV_PLAIN_FP64), dict(precision=g.GCV_MIXED), dict(precision=g.GCV_MIXED, learned=True)]


def once(b, form, graph, stream):
    with torch.cuda.stream(stream):
        arrays, counts, pos = device(b)
        out = torch.empty_like(pos)
        stream.synchronize()
        with g.ArclengthCalculateGpu.from_device_batch(*arrays, rtol=1e-9, stream=stream.cuda_stream, **form) as calc:
            if form.get("learned"):
                calc.set_learned_model(learned.load_model())
            if graph:
                calc.stepGraph(counts, pos, out)
                calc.stepGraph(counts, pos, out)
            else:
                calc.createArclengthTable()
                calc.arclengthReverseInto(counts, pos, out, True, g.GCV_RETURN_US)
            return calc.getAllCurveArclengths().copy(), out.cpu().numpy()


def test_captures_beside_other_threads(gpu_lib):
    batches = [ds.uneven_batch(150, seed=i, max_ctrl=80, max_samples=64) for i in range(3)]
    calls = [(i, f, graph) for i in range(3) for f in range(3) for graph in (False, True)]
    streams = [torch.cuda.Stream() for _ in range(5)]
    want = {c: once(batches[c[0]], FORMS[c[1]], c[2], streams[4]) for c in calls}
    wrong = []

    def work(t):
        order = np.random.default_rng(t).permutation(len(calls))
        for k in order:
            c = calls[k]
            try:
                got = once(batches[c[0]], FORMS[c[1]], c[2], streams[t])
                if not all(np.array_equal(x, y) for x, y in zip(got, want[c])):
                    wrong.append((t, c, "differs"))
            except Exception as e:
                wrong.append((t, c, str(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]

"""Bundle files at the edges of the parser's blocks: tokens across 4 KiB chunks
and longer than the staged halo, records across and longer than the record
walk's window, many small files, a cut-short last record.  Against the host
reader, bit for bit (both convert decimals correctly rounded)."""
import numpy as np
import pytest

import gcurval_gb300 as g
from gcurval_gb300 import bundle

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def text_of(sizes, seed, sep=" "):
    rng = np.random.default_rng(seed)
    out = []
    for nc in sizes:
        nc = int(nc)
        rows = [rng.normal(0, 10, nc), rng.normal(0, 10, nc),
                np.concatenate([np.zeros(4), np.sort(rng.random(nc - 4)), np.ones(4)])]
        out.append("3 %d %d\n" % (nc, nc + 4) + "\n".join(sep.join("%.6g" % v for v in r) for r in rows))
    return "\n".join(out)


def check(texts, tmp_path):
    paths = []
    for i, t in enumerate(texts):
        paths.append(str(tmp_path / f"b{i}"))
        (tmp_path / f"b{i}").write_text(t)
    want = bundle.load(paths)
    got = [a.cpu().numpy() for a in bundle.load_device(paths)]
    for a, b in zip(got, (want.kind, want.degree, want.dim, want.knot_off, want.knots, want.ctrl_off, want.ctrl)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("sizes", [[4], [4] * 400, [1360, 4, 1361, 1362, 4, 5], [5000, 4, 20000, 7], list(range(4, 300))])
def test_record_sizes(sizes, gpu_lib, tmp_path):
    check([text_of(sizes, seed=len(sizes))], tmp_path)


@pytest.mark.parametrize("gap", [1, 63, 64, 65, 4095, 4096, 4097])
def test_blanks_between_numbers(gap, gpu_lib, tmp_path):
    check([text_of([4, 6, 5], seed=gap, sep=" " * gap)], tmp_path)


@pytest.mark.parametrize("zeros", [40, 70, 200, 5000])
def test_long_tokens(zeros, gpu_lib, tmp_path):
    t = text_of([9, 4, 12], seed=zeros)
    check([t.replace(" 0.", " " + "0" * zeros + "0.")], tmp_path)


def test_many_small_files(gpu_lib, tmp_path):
    rng = np.random.default_rng(2)
    check([text_of(rng.integers(4, 13, rng.integers(1, 5)), seed=i) for i in range(70)], tmp_path)


@pytest.mark.parametrize("drop", [1, 2, 5])
@pytest.mark.parametrize("sizes", [[4, 5], [1362, 4], [4] * 500])
def test_cut_short_records_are_rejected(sizes, drop, gpu_lib):
    words = text_of(sizes, seed=1).split()
    with pytest.raises(g.GcvError, match="malformed curve record"):
        bundle.load_device(" ".join(words[:-drop]).encode())

"""Training gradients at the edges of the kernels' tiles and row chunks: row
counts around 64-row tiles, 16-row steps and the point where the chunks grow
beyond 64 rows, and feature rows that are not 16-byte aligned.

Tolerance: FP32 sums over n rows in chunks, against FP64.  The products carry
a few 2^-24 relative each and the sums of K <= 128 terms before them another
factor sqrt(128), about 1e-5 of the layer's gradient norm; 1e-4 is the bar the
other training tests use.
"""
import numpy as np
import pytest

from gcurval_gb300 import learned
from oracle import mlp

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 15, 63, 64, 65, 80, 129, 4095, 4096, 4097, 8200])
def test_gradients(n, offset, gpu_lib):
    rng = np.random.default_rng(n)
    w = (mlp.he_init(3) * 0.5).astype(np.float32)
    X = rng.normal(size=(n, 16)).astype(np.float32)
    depth = rng.integers(0, 13, n).astype(np.int32)
    share = rng.dirichlet(np.ones(4), n).astype(np.float32)
    tg = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    flat = torch.zeros(n * 16 + offset, device="cuda")
    flat[offset:] = torch.from_numpy(X.reshape(-1)).cuda()
    rows = flat[offset:].view(n, 16)
    assert rows.data_ptr() % 16 == 4 * offset
    tr = learned.Trainer(n, weights=w)
    got, loss = tr.gradients(rows, *[torch.from_numpy(a).cuda() for a in (depth, share, tg)])
    again, _ = tr.gradients(rows, *[torch.from_numpy(a).cuda() for a in (depth, share, tg)])
    tr.close()
    np.testing.assert_array_equal(got, again)
    lo, want = mlp.loss_and_grad(w.astype(np.float64), X, depth, share, tg)
    np.testing.assert_allclose(loss, lo, rtol=2e-5)
    o = 0
    for name, shp in mlp.SHAPES:
        k = int(np.prod(shp))
        assert np.linalg.norm(got[o:o + k] - want[o:o + k]) <= 1e-4 * np.linalg.norm(want[o:o + k]) + 1e-7, name
        o += k

"""The training loss is summed in a fixed order: two calls on the same rows give the
same bits, and the mean is as good as the other training tests want it (2e-5)."""
import numpy as np
import pytest

from gcurval_gb300 import learned
from oracle import mlp

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 31, 64, 65, 8192, 50_001])
def test_loss_repeats(n, gpu_lib):
    rng = np.random.default_rng(n)
    w = (mlp.he_init(5) * 0.5).astype(np.float32)
    X = rng.normal(size=(n, 16)).astype(np.float32)
    depth = rng.integers(0, 13, n).astype(np.int32)
    share = rng.dirichlet(np.ones(4), n).astype(np.float32)
    tg = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    rows = [torch.from_numpy(a).cuda() for a in (X, depth, share, tg)]
    tr = learned.Trainer(n, weights=w)
    loss = [tr.gradients(*rows)[1] for _ in range(12)]
    tr.close()
    for other in loss[1:]:
        np.testing.assert_array_equal(other, loss[0])
    want, _ = mlp.loss_and_grad(w.astype(np.float64), X, depth, share, tg)
    np.testing.assert_allclose(loss[0], want, rtol=2e-5)

"""A trainer holds partial gradients for the row chunks of its largest batch, not for
the 64 chunks of a large one (0.16 MB each): 16 trainers of 64 rows take less than
their weights, moments, gradients, activations and one chunk, rounded up to the 2 MB
that the driver hands out.  Batches at the edges of the chunk rule run within it."""
import numpy as np
import pytest

from gcurval_gb300 import learned
from oracle import mlp

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_small_trainers_are_small(gpu_lib):
    learned.Trainer(64).close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    held = [learned.Trainer(64) for _ in range(16)]
    taken = before - torch.cuda.mem_get_info()[0]
    for t in held:
        t.close()
    assert taken <= 16 * 4 << 20


@pytest.mark.parametrize("max_batch", [64, 65, 4096, 4097, 5000])
def test_every_batch_of_a_trainer(max_batch, gpu_lib):
    rng = np.random.default_rng(max_batch)
    w = (mlp.he_init(3) * 0.5).astype(np.float32)
    tr = learned.Trainer(max_batch, weights=w)
    for n in sorted({1, max_batch - 1, max_batch, min(max_batch, 4096)}):
        X = rng.normal(size=(n, 16)).astype(np.float32)
        rows = (X, rng.integers(0, 13, n).astype(np.int32), rng.dirichlet(np.ones(4), n).astype(np.float32),
                rng.uniform(-1, 1, (n, 8)).astype(np.float32))
        got, _ = tr.gradients(*[torch.from_numpy(a).cuda() for a in rows])
        _, want = mlp.loss_and_grad(w.astype(np.float64), *rows)
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
    tr.close()

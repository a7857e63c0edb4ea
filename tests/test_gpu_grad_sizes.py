"""Loss and gradient of the training kernels at batch sizes around their tiles (128 rows, 16-row slices, 16 rows per
head block) against the float64 restatement: float32 sums over the layers' 128 terms and the batch, 1e-5 of the loss
and 1e-4 of the gradient's norm, as for the other batch sizes."""
import numpy as np
import pytest

import mlp_oracle
from code_mpm_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 17, 127, 128, 129, 5000])
def test_loss_and_gradient(n):
    rng = np.random.Generator(np.random.PCG64(n))
    net = engine.Net(n_samples=1000)
    x = np.zeros((n, 16), dtype=np.float32)
    x[:, :13] = rng.normal(0.0, 0.7, (n, 13))
    t = np.zeros((n, 8), dtype=np.float32)
    t[:, :7] = rng.normal(0.0, 1.0, (n, 7))
    loss, grad = net.loss_grad(x, t)
    want_loss, want = mlp_oracle.loss_and_grad(net.params(), x.astype(np.float64), t.astype(np.float64))
    net.close()
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    assert np.linalg.norm(grad - want) <= 1e-4 * np.linalg.norm(want)

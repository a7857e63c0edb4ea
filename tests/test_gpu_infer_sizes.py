"""The tensor-core inference at the edges of its tiles, slots and rounds.

A CTA runs two 128-sample tiles at a time in separate pipelines that carry the inputs, the outputs and the elastic
predictor's strain increments from one round to the next.  Each sample's arithmetic is its own (a row of the operand, a
lane of tensor memory), so a sample's outputs are the same bits wherever it stands: rows of one small set, repeated to
n, give that set's outputs repeated, and nothing past n is written.
"""
import numpy as np
import pytest
import torch

from code_mpm_gb300 import engine
from test_gpu_surrogate import MAT, random_params, samples

pytestmark = pytest.mark.gpu

ROWS = 97
SMS = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 152
ROUND = SMS * 256


@pytest.fixture(scope="module")
def net():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()
    n = engine.Net(**MAT, n_samples=1000)
    n.set_params(random_params(11, scale=2.0))
    return n


def _run(net, x, guard):
    n = x.shape[0]
    out = torch.full((n + guard, 7), float("nan"), dtype=torch.float32, device="cuda")
    net.infer_device(x.data_ptr(), out.data_ptr(), n, engine.INFER_TC)
    torch.cuda.synchronize()
    assert torch.isnan(out[n:]).all()
    return out[:n]


@pytest.mark.parametrize("n", [1, 127, 129, 255, 256, 257, ROUND - 1, ROUND, ROUND + 1, 2 * ROUND + 128,
                               3 * ROUND + 129, 5 * ROUND])
def test_a_samples_place_does_not_matter(net, n):
    rows = torch.tensor(samples(ROWS, seed=3).astype(np.float32), device="cuda").contiguous()
    pick = torch.arange(n, device="cuda") % ROWS
    want = _run(net, rows, 256)
    assert torch.isfinite(want).all()
    got = _run(net, rows[pick].contiguous(), 256)
    assert torch.equal(got, want[pick])

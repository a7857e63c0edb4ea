"""The allocation-free cell order at the sizes where its tiles and its choice of tile size change, against numpy's
stable sort by the IEEE quotient's cell keys (integers: equal)."""
import numpy as np
import pytest

from code_mpm_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 2049, 786_432, 786_433])
@pytest.mark.parametrize("cells", [(3, 2, 1), (70, 60, 50), (300, 200, 100)])  # one, three and three digits
def test_order_equals_a_stable_sort(n, cells):
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(n))
    h = 1.0e-3
    length = tuple(c * h for c in cells)
    pos = rng.uniform(-1.5 * h, 1.02, (3, n)) * np.array(length)[:, None]
    cell = np.array(length) / np.array(cells)
    b = np.floor(pos / cell[:, None])
    kd = np.array(cells, dtype=np.int64) + 2
    key = ((b[0] + 1) + kd[0] * ((b[1] + 1) + kd[1] * (b[2] + 1))).astype(np.int64)
    inside = np.all((b >= -1) & (b <= np.array(cells)[:, None]), axis=0)
    key = np.where(inside, key, kd.prod())
    d = torch.from_numpy(pos).cuda()
    keys = torch.zeros(n, dtype=torch.int32, device="cuda")
    order = torch.zeros(n, dtype=torch.int32, device="cuda")
    assert engine.cell_order_noalloc(length, cells, d.data_ptr(), n, keys.data_ptr(), order.data_ptr()) == 0
    torch.cuda.synchronize()
    assert np.array_equal(keys.cpu().numpy().astype(np.int64), key)
    assert np.array_equal(order.cpu().numpy().astype(np.int64), np.argsort(key, kind="stable"))

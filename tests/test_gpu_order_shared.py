"""The allocation-free cell order given one array for keys and order, by a caller that wants the order alone: equal to
the order of a call with two, with one digit (the first pass reads the keys and writes the order) and with three."""
import numpy as np
import pytest

from code_mpm_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5000, 300_001])
@pytest.mark.parametrize("cells", [(3, 2, 1), (70, 60, 50)])
def test_one_array_for_both(n, cells):
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(n))
    length = tuple(c * 1.0e-3 for c in cells)
    pos = torch.from_numpy(rng.uniform(-0.1, 1.1, (3, n)) * np.array(length)[:, None]).cuda()
    keys, order, both = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
    for k, o in ((keys, order), (both, both)):
        assert engine.cell_order_noalloc(length, cells, pos.data_ptr(), n, k.data_ptr(), o.data_ptr()) == 0
        torch.cuda.synchronize()
    assert np.array_equal(order.cpu().numpy(), np.argsort(keys.cpu().numpy(), kind="stable"))
    assert torch.equal(both, order)

"""Planned thin products where one thread to a row gives way to the tile
kernel: K beyond one stage of the thin operand with fewer than 16384 rows."""
import numpy as np
import pytest
import torch

from launches import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [True, False])
@pytest.mark.parametrize("wide,thin,k,kernel", [(14000, 3, 64, "thin"), (14000, 3, 65, "tile"), (16383, 3, 65, "tile"),
                                                (16384, 3, 65, "thin")])
def test_kernel_and_result(wide, thin, k, kernel, rows):
    from dtcf_gb300.leaves import Group, Triple, MODE_FP64
    m, n = (wide, thin) if rows else (thin, wide)
    rng = np.random.default_rng(wide + k)
    A, B, C = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (m, n))
    a, b, c = (torch.from_numpy(x.copy()).cuda() for x in (A, B, C))
    g = Group([Triple(a.data_ptr(), b.data_ptr(), c.data_ptr(), k, 1, k, 1, n, m, n, k, 0.5, 0)], mode=MODE_FP64)
    names = launches(lambda st: g.execute(stream=st))
    assert any(kernel in name for name, _ in names), names
    torch.cuda.synchronize()
    # one product, numpy's or the kernel's in any order: k + 1 roundings of at most the sum of magnitudes
    bound = 2 * (k + 1) * 2.0 ** -53 * 0.5 * (np.abs(A) @ np.abs(B).T)
    assert np.all(np.abs(c.cpu().numpy() - 0.5 * (A @ B.T)) <= bound)

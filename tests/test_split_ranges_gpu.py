"""Where the split engine cuts K into ranges at two and three slices: products
whose K the accumulators hold twice over run whole, in one launch."""
import numpy as np
import pytest
import torch

from launches import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slices,k,ranges", [(2, 1024, False), (2, 1025, True), (3, 640, False), (3, 641, True),
                                             (4, 512, False), (4, 513, True)])
def test_launches_and_exact_integers(slices, k, ranges):
    """Integers of one digit: the product is the exact one either way."""
    from dtcf_gb300.leaves import Group, Triple, MODE_SPLIT
    m, n = 700, 130
    rng = np.random.default_rng(k)
    A, B = (rng.integers(-127, 128, (x, k)).astype(np.float64) for x in (m, n))
    a, b = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    c = torch.full((m, n), np.nan, dtype=torch.float64, device="cuda")
    g = Group([Triple(a.data_ptr(), b.data_ptr(), c.data_ptr(), k, 1, k, 1, n, m, n, k, 1.0, 0)], mode=MODE_SPLIT,
              slices=slices)
    names = [name for name, _ in launches(lambda st: g.execute(stream=st))]
    assert any("split_reduce" in x for x in names) == ranges, names
    torch.cuda.synchronize()
    assert np.array_equal(c.cpu().numpy(), A @ B.T)

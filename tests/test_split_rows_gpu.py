"""The operand splits at the row lengths where their paths change (lanes per
row, registers or re-read, one CTA or several per row), with rows that start
on and off 16-byte boundaries, zero rows, zero elements and both signs: the
product with a unit matrix gives every element back, rounded to the slices'
step of its row scale."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 7, 15, 16, 17, 31, 32, 33, 63, 64, 65, 128, 255, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4097, 9001,
           16384, 16385, 40001]


def rows_of(rng, m, k):
    x = rng.uniform(-1, 1, (m, k)) * 10.0 ** rng.integers(-3, 4, (m, 1))
    x[rng.random((m, k)) < 0.1] = 0.0
    x[m // 2] = 0.0
    return x


@pytest.mark.parametrize("slices", [2, 4, 6, 7])
@pytest.mark.parametrize("k", LENGTHS)
def test_elements_survive(slices, k):
    """C = A E^T with E rows of one 1: every picked element of A, to half a step 2^(e - F) of its row."""
    from dtcf_gb300.leaves import Group, Triple, MODE_SPLIT
    rng = np.random.default_rng(k + slices)
    m, n = 37, min(k, 40)
    A = rows_of(rng, m, k)
    pick = np.sort(rng.choice(k, n, replace=False))
    pick[-1] = k - 1
    E = np.zeros((n, k))
    E[np.arange(n), pick] = 1.0
    lead = 1 if k % 2 else 0  # an odd stride already moves rows off the boundary; begin there as well
    buf = torch.zeros(m * k + 1, dtype=torch.float64, device="cuda")
    dA = buf[lead:lead + m * k]
    dA.copy_(torch.from_numpy(A.reshape(-1)).cuda())
    dE = torch.from_numpy(E).cuda()
    C = torch.full((m, n), np.nan, dtype=torch.float64, device="cuda")
    t = Triple(dA.data_ptr(), dE.data_ptr(), C.data_ptr(), k, 1, k, 1, n, m, n, k, 1.0, 0)
    g = Group([t], mode=MODE_SPLIT, slices=slices)
    g.execute()
    torch.cuda.synchronize()
    top = np.abs(A).max(axis=1, keepdims=True)
    e = np.where(top > 0, np.frexp(np.where(top > 0, top, 1.0))[1], 0)
    step = np.where(top > 0, np.ldexp(1.0, e - (7 + 8 * (slices - 1))), 0.0)
    got = C.cpu().numpy()
    assert np.all(np.abs(got - A[:, pick]) <= step / 2 + 2.0 ** -52 * np.abs(A[:, pick]))
    assert not got[m // 2].any()

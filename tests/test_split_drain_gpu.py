"""The ends of a split GEMM's tiles: sums made FP64 values by integer
instructions, in vector stores where rows allow them, and the way round both
near the ends of the FP64 range.  Integers that the leading slices hold, rows
and columns scaled by powers of two: every result is exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# bits whose digits fill so many leading slices that no kept product is missing
BITS = {2: 7, 3: 15, 4: 15, 5: 20, 6: 20, 7: 20}


def product(A, B, slices, lead, ld):
    """A B^T into a buffer from element lead on, rows ld apart."""
    from dtcf_gb300.leaves import Group, Triple, MODE_SPLIT
    (m, k), n = A.shape, B.shape[0]
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    buf = torch.full((lead + m * ld + 8,), np.nan, dtype=torch.float64, device="cuda")
    g = Group([Triple(dA.data_ptr(), dB.data_ptr(), buf.data_ptr() + 8 * lead, k, 1, k, 1, ld, m, n, k, 1.0, 0)],
              mode=MODE_SPLIT, slices=slices)
    g.execute()
    torch.cuda.synchronize()
    out = buf.cpu().numpy()
    rows = out[lead:lead + m * ld].reshape(m, ld)
    assert np.isnan(out[:lead]).all() and np.isnan(rows[:, n:]).all() and np.isnan(out[lead + m * ld:]).all()
    return rows[:, :n]


@pytest.mark.parametrize("slices", sorted(BITS))
@pytest.mark.parametrize("lead,pad", [(0, 0), (1, 0), (2, 2), (4, 4), (0, 1)])
@pytest.mark.parametrize("m,n,k", [(130, 6, 40), (70, 31, 64), (33, 32, 17), (130, 64, 70), (40, 33, 300), (129, 100, 65)])
def test_scales_and_strides(slices, lead, pad, m, n, k):
    rng = np.random.default_rng(slices + 10 * lead + m + n)
    top = 1 << BITS[slices]
    A = rng.integers(-top + 1, top, (m, k)).astype(np.float64)
    B = rng.integers(-top + 1, top, (n, k)).astype(np.float64)
    A[m // 3] = 0.0
    B[n // 2] = 0.0
    # 32 rows of ordinary scale, 32 of mixed, then the ends of the range
    p = rng.integers(-40, 41, m)
    p[32:64] = rng.choice([-880, 0, 880], len(p[32:64]))
    p[64:] = rng.choice([-900, 900], len(p[64:]))
    q = rng.choice([-30, 0, 30], n)
    got = product(np.ldexp(A, p[:, None]), np.ldexp(B, q[:, None]), slices, lead, n + pad)
    want = np.ldexp((A.astype(np.int64) @ B.astype(np.int64).T).astype(np.float64), p[:, None] + q[None, :])
    assert np.array_equal(got, want)


@pytest.mark.parametrize("slices", [4, 5, 6])
@pytest.mark.parametrize("k", [32767, 32768, 32769, 70001])
@pytest.mark.parametrize("n", [1, 70])
def test_long_rows(slices, k, n):
    rng = np.random.default_rng(slices + k)
    top = 1 << min(BITS[slices], 17)
    A, B = rng.integers(0, top, (5, k)).astype(np.float64), rng.integers(0, top, (n, k)).astype(np.float64)
    got = product(A, B, slices, 0, n)
    assert np.array_equal(got, (A.astype(np.int64) @ B.astype(np.int64).T).astype(np.float64))

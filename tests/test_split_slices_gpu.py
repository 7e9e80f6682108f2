"""The k-stationary split kernel at every slice count where its accumulator
groups begin and end: K around one k-block, one group of the high levels, one
of the low ones and several of both, ragged tiles, and K long enough to be
cut into ranges.  On integers that the leading slices hold, the products kept
are all there are, so the result is the exact integer product; on random data
the error stays below the slices' bound."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# bits whose digits fill so many leading slices that no kept product is missing: s + t <= S + 1
BITS = {2: 7, 3: 15, 4: 15, 5: 20, 6: 20, 7: 20}


@pytest.mark.parametrize("slices", sorted(BITS))
@pytest.mark.parametrize("M,N,K", [(129, 65, 65), (128, 64, 160), (130, 40, 161), (200, 200, 257), (64, 33, 513),
                                   (300, 130, 1100), (17, 90, 9000)])
def test_exact_on_integers(slices, M, N, K):
    import dtcf_gb300
    rng = np.random.default_rng(slices * K + M)
    top = 1 << BITS[slices]
    A = rng.integers(-top + 1, top, size=(M, K)).astype(np.float64)
    B = rng.integers(-top + 1, top, size=(N, K)).astype(np.float64)
    C = torch.full((M, N), np.nan, dtype=torch.float64, device="cuda")
    dtcf_gb300.split_gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C, slices=slices)
    want = (A.astype(np.int64) @ B.astype(np.int64).T).astype(np.float64)
    assert np.array_equal(C.cpu().numpy(), want)


@pytest.mark.parametrize("slices", sorted(BITS))
def test_error_bound_on_random_rows(slices):
    """Each operand keeps 7 + 8 (S - 1) bits below its row's scale (|x| < 2^e, e <= 0 here), and the products dropped
    weigh below S 2^-(8 S - 2) (1 + 2^-7): together under (S + 4) 2^(2 - 8 S) per element."""
    import dtcf_gb300
    rng = np.random.default_rng(slices)
    M, N, K = 200, 100, 2000
    A, B = rng.uniform(-1, 1, (M, K)), rng.uniform(-1, 1, (N, K))
    C = torch.zeros((M, N), dtype=torch.float64, device="cuda")
    dtcf_gb300.split_gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C, slices=slices)
    want = np.asarray(A, dtype=np.longdouble) @ np.asarray(B, dtype=np.longdouble).T
    bound = K * ((slices + 4) * 2.0 ** (2 - 8 * slices)) + 2.0 ** -51 * np.abs(want).max()
    assert np.max(np.abs(C.cpu().numpy() - want)) <= bound

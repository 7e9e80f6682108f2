"""The FP64 tile kernel's schedules -- a tile per warp, per CTA and per
cluster, K cut into ranges, ragged edges in every direction -- against numpy
on all four operand orders, and the grouped form against the one-call form."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# K > 8 (shorter K has its own kernel); comments name what each size reaches
SHAPES = [
    (1, 1, 9), (8, 8, 12), (9, 7, 13), (16, 16, 16),  # one tile, whole and ragged, K not a multiple of 4
    (64, 48, 96), (17, 33, 65),                       # 8 x 8 tiles, clusters
    (24, 24, 3456), (5, 3, 20000),                    # few outputs: clusters of 8, K ranges
    (300, 290, 77), (700, 650, 30),                   # 16 x 16 tiles per CTA
    (8000, 200, 9), (31, 9000, 21),                   # a tile per warp; thin on the other side
]


def _operands(m, n, k, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (m, n))


def _bound(A, B, C, alpha):
    """Any order of k products and sums, numpy's and the kernel's: (k + 2) roundings each of at most the sum of
    magnitudes."""
    k = A.shape[1]
    return 2 * (k + 2) * 2.0 ** -53 * (np.abs(alpha) * (np.abs(A) @ np.abs(B).T) + np.abs(C))


@pytest.mark.parametrize("at,bt", [(0, 1), (1, 0), (0, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_one_call(m, n, k, at, bt):
    import dtcf_gb300 as gbx
    A, B, C = _operands(m, n, k, m + n + k)
    dA = torch.from_numpy(np.ascontiguousarray(A.T if at else A)).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B if bt else B.T)).cuda()
    dC = torch.from_numpy(C.copy()).cuda()
    gbx.local_contraction(m, n, k, dA, dB, dC, at, bt, -0.75)
    got = dC.cpu().numpy()
    assert np.all(np.abs(got - (C - 0.75 * (A @ B.T))) <= _bound(A, B, C, 0.75))


def test_grouped_shapes_share_a_launch():
    """All shapes in one planned set: each problem's tiles, K ranges and edges beside the others'."""
    from dtcf_gb300.leaves import Group, Triple, MODE_FP64
    data = [_operands(m, n, k, 3 * m + n + k) for m, n, k in SHAPES]
    dev = [[torch.from_numpy(x.copy()).cuda() for x in t] for t in data]
    tri = [Triple(a.data_ptr(), b.data_ptr(), c.data_ptr(), k, 1, k, 1, n, m, n, k, 0.5, i % 2)
           for i, ((m, n, k), (a, b, c)) in enumerate(zip(SHAPES, dev))]
    Group(tri, mode=MODE_FP64).execute()
    torch.cuda.synchronize()
    for i, ((A, B, C), (_, _, c)) in enumerate(zip(data, dev)):
        C = C if i % 2 else 0 * C
        assert np.all(np.abs(c.cpu().numpy() - (C + 0.5 * (A @ B.T))) <= _bound(A, B, C, 0.5)), SHAPES[i]

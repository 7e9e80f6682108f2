"""Short steps at the sizes where their work is divided differently: operand
splits by a warp or a CTA to a row (the row count and row length at which they
change), both operands' packs in one launch (small and large sets of moves,
in either place, odd and even tiles), and products formed in place whose items
are smaller than a CTA, end inside one, or cover several passes."""
import numpy as np
import pytest
import torch

import oracle.rrr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slices", [3, 6])
@pytest.mark.parametrize("rows", [1215, 1216, 1217, 2500])
@pytest.mark.parametrize("k", [128, 129, 401, 1024, 1025])
def test_row_counts(slices, rows, k):
    """rows rows of both operands together: every element of A comes back from a product with unit rows, to half a
    step 2^(e - F) of its row's scale."""
    from dtcf_gb300.leaves import Group, Triple, MODE_SPLIT
    rng = np.random.default_rng(rows + k + slices)
    n = 24
    m = rows - n
    A = rng.uniform(-1, 1, (m, k)) * 10.0 ** rng.integers(-3, 4, (m, 1))
    A[m // 2] = 0.0
    pick = np.sort(rng.choice(k, n, replace=False))
    pick[-1] = k - 1
    E = np.zeros((n, k))
    E[np.arange(n), pick] = 1.0
    dA, dE = torch.from_numpy(A).cuda(), torch.from_numpy(E).cuda()
    C = torch.full((m, n), np.nan, dtype=torch.float64, device="cuda")
    g = Group([Triple(dA.data_ptr(), dE.data_ptr(), C.data_ptr(), k, 1, k, 1, n, m, n, k, 1.0, 0)], mode=MODE_SPLIT,
              slices=slices)
    g.execute()
    torch.cuda.synchronize()
    top = np.abs(A).max(axis=1, keepdims=True)
    e = np.where(top > 0, np.frexp(np.where(top > 0, top, 1.0))[1], 0)
    step = np.where(top > 0, np.ldexp(1.0, e - (7 + 8 * (slices - 1))), 0.0)
    got = C.cpu().numpy()
    assert np.all(np.abs(got - A[:, pick]) <= step / 2 + 2.0 ** -52 * np.abs(A[:, pick]))
    assert not got[m // 2].any()


def make(size, blk, rng):
    from dtcf_gb300.rrr import Tensor
    t = Tensor("cccc"[:len(size)], size, tuple(s // b for s, b in zip(size, blk)))
    t.tiles.copy_(torch.from_numpy(rng.uniform(-1, 1, t.tiles.numel())).cuda())
    return t


def as_oracle(t):
    return dict(tiles=t.tiles.cpu().numpy().reshape(t.num_tiles, -1), addrs=t.addrs, sym=t.sym,
                block_range=t.block_range, vgrid=t.vgrid)


@pytest.mark.parametrize("mode", ["fp64", "split"])
@pytest.mark.parametrize("big", [0, 1, 2])
@pytest.mark.parametrize("b", [5, 8])
def test_packs(mode, big, b):
    """C[a,b,i,j] += alpha A[a,e,i,m] B[e,b,m,j], K = 100 or more; big: the operand whose pack is cut into large chunks."""
    from dtcf_gb300.rrr import Contraction
    rng = np.random.default_rng(b + 10 * big)
    a, c = ((4, 1), (1, 4), (4, 4))[big]
    e = 4
    size = lambda w: tuple(x * b for x in w)  # noqa: E731
    blk = (b,) * 4
    A, B = make(size((a, e, a, e)), blk, rng), make(size((e, c, e, c)), blk, rng)
    C = make(size((a, c, a, c)), blk, rng)
    ops = [as_oracle(t) for t in (A, B, C)]
    want = oracle.rrr.contract(*ops, "a,e,i,m", "e,b,m,j", "a,b,i,j", 0.5, 1)
    K = (e * b) ** 2
    bound = (2.0 ** -53 * (K + 4) if mode == "fp64" else 2.0 ** -44) * 0.5 * K + 2.0 ** -50 * np.abs(want).max()
    Contraction(A, B, C, mode=mode, sign=1).contract("a,e,i,m", "e,b,m,j", "a,b,i,j", 0.5)
    torch.cuda.synchronize()
    assert np.max(np.abs(C.tiles.cpu().numpy().reshape(want.shape) - want)) <= bound


@pytest.mark.parametrize("tiles", [(1, 1, 1, 1), (1, 2, 3, 1), (4, 3, 3, 2)])
@pytest.mark.parametrize("blk", [(1, 1, 1, 1), (4, 4, 8, 4), (5, 3, 7, 5), (8, 8, 8, 4), (7, 9, 11, 3), (13, 12, 11, 10)])
def test_products_in_place(tiles, blk):
    """C[a,b,i,j] += alpha F[a,e] T[e,b,i,j] with a short contracted index: tiles of 1 to 17160 elements."""
    from dtcf_gb300.rrr import Contraction
    rng = np.random.default_rng(sum(blk) + sum(tiles))
    size = tuple(t * x for t, x in zip(tiles, blk))
    F = make((size[0], size[0]), (blk[0], blk[0]), rng)
    T, C = make(size, blk, rng), make(size, blk, rng)
    ops = [as_oracle(t) for t in (F, T, C)]
    want = oracle.rrr.contract(*ops, "a,e", "e,b,i,j", "a,b,i,j", 0.5, 1)
    bound = 2.0 ** -53 * (size[0] + 4) * 0.5 * size[0] + 2.0 ** -50 * np.abs(want).max()
    Contraction(F, T, C, mode="fp64", sign=1).contract("a,e", "e,b,i,j", "a,b,i,j", 0.5)
    torch.cuda.synchronize()
    assert np.max(np.abs(C.tiles.cpu().numpy().reshape(want.shape) - want)) <= bound

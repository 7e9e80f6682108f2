"""One-call permutes and packs where their boxes, tables and edges change:
extents around the box runs, every route (straight, staged, cut boxes, many
permutations in one call, more blocks and tiles than one launch's tables
hold), bit for bit against numpy."""
import itertools
import random

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64).reshape(-1)).cuda()


def permuted(x, perm):
    inv = [0] * len(perm)
    for i, p in enumerate(perm):
        inv[p] = i
    return np.ascontiguousarray(x.transpose(inv)).reshape(-1)


WIDTHS = [(1,), (5000,), (1, 1, 1), (129, 257), (4097, 3), (3, 4097), (2, 2, 2, 2, 2, 2, 2, 2), (3, 5, 2, 3, 4, 3, 2, 5),
          (64, 64, 64), (17, 1, 33, 65), (13, 40, 7, 31), (2, 3, 5000), (5000, 3, 2), (31, 8, 8, 47), (1, 700, 1, 900)]


@pytest.mark.parametrize("widths", WIDTHS)
def test_transpose(widths):
    import dtcf_gb300 as gbx
    rng = random.Random(str(widths))
    x = np.random.default_rng(len(widths)).uniform(-1, 1, widths)
    d = dev(x)
    perms = {tuple(range(len(widths))), tuple(reversed(range(len(widths))))}
    perms |= {tuple(rng.sample(range(len(widths)), len(widths))) for _ in range(6)}
    for p in perms:
        y = torch.full_like(d, np.nan)
        gbx.transpose(d, y, p, widths)
        assert np.array_equal(y.cpu().numpy(), permuted(x, p)), p


@pytest.mark.parametrize("widths,count,nperm", [((4, 4, 4, 4), 5000, 24), ((2, 2, 2, 2), 40000, 8), ((5, 3, 7, 2), 2049, 24),
                                                ((16, 16, 9, 9), 40, 3), ((30, 2, 70, 3), 7, 5), ((6, 6, 6), 3000, 1)])
def test_transpose_blocks(widths, count, nperm):
    """Blocks of up to 24 permutations (more than one launch carries) and more blocks than a launch's table."""
    import dtcf_gb300 as gbx
    rng = random.Random(count)
    all_p = list(itertools.permutations(range(len(widths))))
    choice = rng.sample(all_p, min(nperm, len(all_p)))
    perms = [choice[0 if nperm > 16 and b < 20 else rng.randrange(len(choice))] for b in range(count)]
    x = np.random.default_rng(count).uniform(-1, 1, (count,) + widths)
    d = dev(x)
    y = torch.full_like(d, np.nan)
    gbx.transpose_blocks(d, y, perms, widths)
    want = np.concatenate([permuted(b, p) for b, p in zip(x, perms)])
    assert np.array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("grid,rpb,cpb", [((2, 3, 2, 2), 5, 7), ((1, 1), 1, 1), ((9, 10, 10, 9), 3, 4), ((3, 2, 4), 70, 66),
                                          ((20, 20, 20), 2, 3)])
@pytest.mark.parametrize("offset", [0, 1])
def test_pack_and_unpack(grid, rpb, cpb, offset):
    """Odd and even tile widths, bases off a 16-byte boundary, more tiles than a launch's table."""
    import dtcf_gb300 as gbx
    addr = list(itertools.product(*[range(g) for g in grid]))
    random.Random(rpb).shuffle(addr)
    nr = len(grid) // 2
    tiles = np.random.default_rng(cpb).uniform(-1, 1, (len(addr), rpb, cpb))
    n = tiles.size
    src, big, back = (torch.full((n + 1,), np.nan, dtype=torch.float64, device="cuda")[offset:offset + n] for _ in range(3))
    src.copy_(dev(tiles))
    rows, cols = gbx.create_big_matrix(grid, list(range(len(grid))), src, addr, rpb, cpb, nr, big)
    assert (rows, cols) == (int(np.prod(grid[:nr])), int(np.prod(grid[nr:])))
    want = np.empty((rows, cols, rpb, cpb))
    for a, t in zip(addr, tiles):
        want[np.ravel_multi_index(a[:nr], grid[:nr]), np.ravel_multi_index(a[nr:], grid[nr:])] = t
    assert np.array_equal(big.cpu().numpy(), want.transpose(0, 2, 1, 3).reshape(-1))
    gbx.revert_big_matrix(grid, list(range(len(grid))), addr, rpb, cpb, nr, big, back)
    assert np.array_equal(back.cpu().numpy(), tiles.reshape(-1))
    # addresses outside the grid still order by rank; a repeated address keeps its first tile
    if len(grid) == 2:
        y = torch.full((3,), np.nan, dtype=torch.float64, device="cuda")
        assert gbx.create_big_matrix([1, 1], [0, 1], dev([1.0, 2.0, 3.0]), [[5, 0], [2, 0], [5, 0]], 1, 1, 1, y) == (2, 1)
        assert y.cpu().numpy()[:2].tolist() == [2.0, 1.0]

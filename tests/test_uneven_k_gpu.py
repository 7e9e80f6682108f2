"""FP64 products of long K beside so many short ones that those take a tile to
a warp: the long ones have a launch of their own, with their K shared."""
import numpy as np
import pytest
import torch

from launches import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("long_shapes,launched", [
    ([(40, 33, 20000)], 2), ([(8, 8, 20001), (16, 200, 9000), (300, 5, 12345)], 2), ([(32, 32, 64)], 1), ([], 1),
])
def test_launches_and_results(long_shapes, launched):
    from dtcf_gb300.leaves import Group, Triple, MODE_FP64
    rng = np.random.default_rng(len(long_shapes))
    shapes = [(32, 32, 32)] * 1500 + long_shapes + [(32, 32, 32)] * 1500
    data, dev, tri = {}, [], []
    for i, s in enumerate(shapes):
        m, n, k = s
        if s not in data:
            A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k))
            data[s] = (A, B, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda())
        c = torch.full((m, n), np.nan, dtype=torch.float64, device="cuda")
        dev.append(c)
        tri.append(Triple(data[s][2].data_ptr(), data[s][3].data_ptr(), c.data_ptr(), k, 1, k, 1, n, m, n, k, 0.5, 0))
    g = Group(tri, mode=MODE_FP64)
    names = [name for name, _ in launches(lambda st: g.execute(stream=st)) if "tile" in name]
    assert len(names) == launched, names
    for per_triple in (False, True):
        for c in dev:
            c.fill_(np.nan)
        g.execute(per_triple=per_triple)
        torch.cuda.synchronize()
        for s, c in zip(shapes, dev):
            A, B, k = data[s][0], data[s][1], s[2]
            # one product, numpy's or the kernel's in any order: k + 1 roundings of at most the sum of magnitudes
            bound = 2 * (k + 1) * 2.0 ** -53 * 0.5 * (np.abs(A) @ np.abs(B).T)
            assert np.all(np.abs(c.cpu().numpy() - 0.5 * (A @ B.T)) <= bound), s


@pytest.mark.parametrize("m,n,k,ctas,reduced", [
    (32, 32, 100000, 304, True),   # K ranges without clusters: two CTAs to every SM
    (100, 100, 50000, 608, True),  # 169 tiles, a few more than SMs
    (28, 3, 17508, 96, True),      # four tiles
    (17, 40, 30001, 120, False), (24, 24, 3456, 72, False), (48, 48, 1500, 288, False),  # clusters, K whole
])
def test_one_long_product(m, n, k, ctas, reduced):
    """A product of few tiles: every SM has work, and its K is cut into ranges where that pays."""
    from dtcf_gb300.leaves import Group, Triple, MODE_FP64
    rng = np.random.default_rng(k)
    A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k))
    a, b = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    c = torch.full((m, n), np.nan, dtype=torch.float64, device="cuda")
    g = Group([Triple(a.data_ptr(), b.data_ptr(), c.data_ptr(), k, 1, k, 1, n, m, n, k, 0.5, 0)], mode=MODE_FP64)
    made = launches(lambda st: g.execute(stream=st))
    assert [x for name, x in made if "tile" in name][0] >= ctas, made
    assert any("reduce" in name for name, _ in made) == reduced, made
    torch.cuda.synchronize()
    bound = 2 * (k + 1) * 2.0 ** -53 * 0.5 * (np.abs(A) @ np.abs(B).T)
    assert np.all(np.abs(c.cpu().numpy() - 0.5 * (A @ B.T)) <= bound)

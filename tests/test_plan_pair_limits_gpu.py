"""FP64 plans over a contracted pair of symmetric indices at the ends of the
FP64 range: small integers times powers of two whose products and sums are
exact, so the result has to be the exact one.  Also the shapes at which the
columns that count twice end inside a K step, a warp's share or a K range."""
import numpy as np
import pytest
import torch

import oracle.rrr

pytestmark = pytest.mark.gpu


def make(sym, size, vgrid, values):
    from dtcf_gb300.rrr import Tensor
    t = Tensor(sym, size, vgrid)
    t.tiles.copy_(torch.from_numpy(values(t.tiles.numel())).cuda())
    return t


def as_oracle(t):
    return dict(tiles=t.tiles.cpu().numpy().reshape(t.num_tiles, -1), addrs=t.addrs, sym=t.sym,
                block_range=t.block_range, vgrid=t.vgrid)


def result(A, B, C, alpha, sign=1):
    from dtcf_gb300.rrr import Contraction
    want = oracle.rrr.contract(as_oracle(A), as_oracle(B), as_oracle(C), "a,b,e,f", "e,f,i,j", "a,b,i,j", alpha, sign)
    Contraction(A, B, C, mode="fp64", sign=sign).contract("a,b,e,f", "e,f,i,j", "a,b,i,j", alpha)
    torch.cuda.synchronize()
    return C.tiles.cpu().numpy().reshape(want.shape), want


@pytest.mark.parametrize("ea,eb,alpha", [
    (-1074, 1000, 1.0),          # odd multiples of the smallest number
    (1000, -1074, 1.0),
    (-540, -530, 1.0),           # sums among the subnormal numbers
    (1019, -1000, 1.0),
    (-300, -700, 2.0 ** 1023),   # a factor that twice it would overflow
    (-300, -700, -1.5 * 2.0 ** 1023),
])
def test_exact_at_the_ends(ea, eb, alpha):
    rng = np.random.default_rng(abs(ea))
    n, g = 24, 3

    def ints(e):
        return lambda k: np.ldexp(rng.integers(1, 8, k).astype(np.float64), e)

    A = make("aabb", (n,) * 4, (g,) * 4, ints(ea))
    B = make("aabb", (n, n, 16, 16), (g, g, 2, 2), ints(eb))
    C = make("aabb", (n, n, 16, 16), (g, g, 2, 2), lambda k: np.zeros(k))
    got, want = result(A, B, C, alpha)
    assert np.all(np.isfinite(want)) and want.all()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("v,vb,o,ob", [(6, 3, 6, 3), (10, 5, 10, 5), (21, 7, 7, 7), (33, 11, 11, 11), (65, 13, 5, 5),
                                       (48, 8, 16, 8), (90, 10, 10, 10), (45, 9, 1, 1), (8, 1, 9, 1)])
def test_exact_integers(v, vb, o, ob):
    """Block pairs of every remainder by four, from one tile to several to an SM, and thin outputs."""
    rng = np.random.default_rng(v)

    def ints(k):
        return rng.integers(-9, 10, k).astype(np.float64)

    A = make("aabb", (v,) * 4, (v // vb,) * 4, ints)
    B = make("aabb", (v, v, o, o), (v // vb, v // vb, o // ob, o // ob), ints)
    C = make("aabb", (v, v, o, o), (v // vb, v // vb, o // ob, o // ob), ints)
    got, want = result(A, B, C, 2.0, -1)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("kernel,ta,tb,tc", [
    # (symmetry, extents, block extents, indices) of A, B and C
    ("gemv", ("aabb", (45,) * 4, (9,) * 4, "a,b,e,f"), ("aacc", (45, 45, 1, 1), (9, 9, 1, 1), "e,f,i,j"),
     ("aacc", (45, 45, 1, 1), (9, 9, 1, 1), "a,b,i,j")),
    ("gemv", ("aac", (33, 33, 2), (11, 11, 2), "e,f,i"), ("aacc", (33, 33, 10, 20), (11, 11, 10, 20), "e,f,j,k"),
     ("ccc", (2, 10, 20), (2, 10, 20), "i,j,k")),
    ("small_out", ("aacc", (28, 28, 22, 9), (7, 7, 11, 9), "e,f,g,i"), ("aacc", (28, 28, 22, 13), (7, 7, 11, 13), "e,f,g,j"),
     ("cc", (9, 13), (9, 13), "i,j")),
    ("thin", ("ccaa", (150, 150, 10, 10), (50, 50, 5, 5), "a,b,e,f"), ("aac", (10, 10, 5), (5, 5, 5), "e,f,i"),
     ("ccc", (150, 150, 5), (50, 50, 5), "a,b,i")),
    ("thin", ("aac", (10, 10, 5), (5, 5, 5), "e,f,i"), ("aacc", (10, 10, 150, 150), (5, 5, 50, 50), "e,f,a,b"),
     ("ccc", (5, 150, 150), (5, 50, 50), "i,a,b")),
])
def test_every_kernel_counts_twice(kernel, ta, tb, tc):
    """The thin kernels too run over block pairs x >= y, at half the products, with exact sums."""
    from dtcf_gb300.rrr import Plan
    from launches import launches
    rng = np.random.default_rng(len(kernel))
    A, B, C = (make(s, size, tuple(n // b for n, b in zip(size, blk)), lambda k: rng.integers(-9, 10, k).astype(np.float64))
               for s, size, blk, _ in (ta, tb, tc))
    names = [t[3] for t in (ta, tb, tc)]
    want = oracle.rrr.contract(as_oracle(A), as_oracle(B), as_oracle(C), *names, 2.0, -1)
    start = C.tiles.clone()
    plan = Plan(A, B, C, *names, mode="fp64", sign=-1)
    made = launches(lambda st: plan.execute(A, B, C, 2.0, stream=st))
    assert any(kernel in name for name, _ in made), made
    torch.cuda.synchronize()
    C.tiles.copy_(start)
    plan.execute(A, B, C, 2.0)
    torch.cuda.synchronize()
    assert np.array_equal(C.tiles.cpu().numpy().reshape(want.shape), want)
    assert np.abs(want - start.cpu().numpy().reshape(want.shape)).max() > 0

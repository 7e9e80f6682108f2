"""Plans over a contracted pair of symmetric indices (run over block pairs
x >= y) against the dense oracle: both signs, either label order, engines,
pairs that do not qualify (a tensor that also stores a flipped block, a
larger group, indices of different groups), missing tiles, and values at the
ends of the FP64 range."""
import numpy as np
import pytest
import torch

import oracle.rrr

pytestmark = pytest.mark.gpu


def make(sym, size, vgrid, rng, addrs=None, scale=1.0):
    from dtcf_gb300.rrr import Tensor
    t = Tensor(sym, size, vgrid, addrs=addrs)
    t.tiles.copy_(torch.from_numpy(rng.uniform(-1, 1, t.tiles.numel()) * scale).cuda())
    return t


def as_oracle(t):
    return dict(tiles=t.tiles.cpu().numpy().reshape(t.num_tiles, -1), addrs=t.addrs, sym=t.sym,
                block_range=t.block_range, vgrid=t.vgrid)


def run(A, B, C, ia, ib, ic, mode, sign, alpha=0.5):
    """(result, oracle's, bound): K products in any order, each of at most max |A| max |B|; the split engine's
    slices (6: 47 bits of the row scale) on top."""
    from dtcf_gb300.rrr import Contraction
    a, b = as_oracle(A), as_oracle(B)
    want = oracle.rrr.contract(a, b, as_oracle(C), ia, ib, ic, alpha, sign)
    K = np.prod([A.size[i] for i, l in enumerate(ia.split(",")) if l in ib.split(",")])
    scale = abs(alpha) * np.abs(a["tiles"]).max() * np.abs(b["tiles"]).max() * K
    bound = (2.0 ** -53 * (K + 4) if mode == "fp64" else 2.0 ** -44) * scale + 2.0 ** -50 * np.abs(want).max()
    Contraction(A, B, C, mode=mode, sign=sign).contract(ia, ib, ic, alpha)
    torch.cuda.synchronize()
    return C.tiles.cpu().numpy().reshape(want.shape), want, bound


@pytest.mark.parametrize("mode", ["fp64", "split"])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("ib", ["e,f,i,j", "f,e,i,j"])
@pytest.mark.parametrize("n,blk", [(24, 8), (25, 5), (6, 6)])
def test_ladder(mode, sign, ib, n, blk):
    rng = np.random.default_rng(n + blk)
    g, o = n // blk, 2
    A = make("aabb", (n,) * 4, (g,) * 4, rng)
    B = make("aabb", (n, n, o * blk, o * blk), (g, g, o, o), rng)
    C = make("aabb", (n, n, o * blk, o * blk), (g, g, o, o), rng)
    got, want, bound = run(A, B, C, "a,b,e,f", ib, "a,b,i,j", mode, sign)
    assert np.max(np.abs(got - want)) <= bound


@pytest.mark.parametrize("mode", ["fp64", "split"])
def test_pairs_that_do_not_qualify(mode):
    rng = np.random.default_rng(7)
    n, blk, g = 24, 8, 3
    B = make("aabb", (n, n, 16, 16), (g, g, 2, 2), rng)
    # A stores a flipped block beside its canonical one: its value is its own
    full = [(a, b, e, f) for a in range(g) for b in range(a + 1) for e in range(g) for f in range(e + 1)]
    A = make("aabb", (n,) * 4, (g,) * 4, rng, addrs=full + [(1, 0, 0, 2)])
    C = make("aabb", (n, n, 16, 16), (g, g, 2, 2), rng)
    got, want, bound = run(A, B, C, "a,b,e,f", "e,f,i,j", "a,b,i,j", mode, -1)
    assert np.max(np.abs(got - want)) <= bound
    # contracted indices of different groups in A; of none in B
    A = make("abab", (n,) * 4, (g,) * 4, rng)
    C = make("cccc", (n, n, 16, 16), (g, g, 2, 2), rng)
    got, want, bound = run(A, make("cccc", (n, n, 16, 16), (g, g, 2, 2), rng), C, "a,b,e,f", "e,f,i,j", "a,b,i,j", mode, -1)
    assert np.max(np.abs(got - want)) <= bound
    # a group of three indices in A
    A3 = make("caaa", (n,) * 4, (g,) * 4, rng)
    C3 = make("cccc", (n, n, 16, 16), (g, g, 2, 2), rng)
    got, want, bound = run(A3, B, C3, "a,b,e,f", "e,f,i,j", "a,b,i,j", mode, 1)
    assert np.max(np.abs(got - want)) <= bound


@pytest.mark.parametrize("mode", ["fp64", "split"])
def test_missing_tiles(mode):
    rng = np.random.default_rng(11)
    n, g = 24, 3
    some = [(a, b, e, f) for a in range(g) for b in range(a + 1) for e in range(g) for f in range(e + 1)
            if (a + b + e + f) % 2 == 0]
    A = make("aabb", (n,) * 4, (g,) * 4, rng, addrs=some)
    B = make("aabb", (n, n, 16, 16), (g, g, 2, 2), rng)
    C = make("aabb", (n, n, 16, 16), (g, g, 2, 2), rng)
    got, want, bound = run(A, B, C, "a,b,e,f", "e,f,i,j", "a,b,i,j", mode, -1)
    assert np.max(np.abs(got - want)) <= bound


@pytest.mark.parametrize("scale", [2.0 ** 1000, 2.0 ** -1000])
def test_extreme_values(scale):
    """Large A against small B: nothing packed may overflow or lose bits."""
    rng = np.random.default_rng(13)
    n, g = 24, 3
    A = make("aabb", (n,) * 4, (g,) * 4, rng, scale=scale)
    B = make("aabb", (n, n, 16, 16), (g, g, 2, 2), rng, scale=1.0 / scale)
    C = make("aabb", (n, n, 16, 16), (g, g, 2, 2), rng)
    got, want, bound = run(A, B, C, "a,b,e,f", "e,f,i,j", "a,b,i,j", "fp64", -1)
    assert np.max(np.abs(got - want)) <= bound


@pytest.mark.parametrize("slices,width", [(4, 0), (5, 0), (6, 0), (7, 0), (6, 32), (6, 128), (4, 256)])
def test_doubled_digits_are_exact(slices, width):
    """Integers of one leading digit near its maximum, all of one sign, so that every accumulator comes as close to
    2^24 as it can: the split engine's result is the exact integer one."""
    from dtcf_gb300._lib import lib
    rng = np.random.default_rng(slices + width)
    n, g = 48, 6
    A, B, C = (make("aabb", s, v, rng) for s, v in (((n,) * 4, (g,) * 4), ((n, n, 16, 16), (g, g, 2, 2)),
                                                   ((n, n, 16, 16), (g, g, 2, 2))))
    for t in (A, B):
        t.tiles.copy_(torch.from_numpy(rng.integers(100, 128, t.tiles.numel()).astype(np.float64)).cuda())
    C.tiles.zero_()
    from dtcf_gb300.rrr import Plan
    want = oracle.rrr.contract(as_oracle(A), as_oracle(B), as_oracle(C), "a,b,e,f", "e,f,i,j", "a,b,i,j", 1.0, 1)
    assert lib().gbx_split_set_width(width) == 0
    try:
        plan = Plan(A, B, C, "a,b,e,f", "e,f,i,j", "a,b,i,j", mode="split", sign=1, slices=slices)
    finally:
        lib().gbx_split_set_width(0)
    plan.execute(A, B, C, 1.0)
    torch.cuda.synchronize()
    assert np.array_equal(C.tiles.cpu().numpy().reshape(want.shape), want)

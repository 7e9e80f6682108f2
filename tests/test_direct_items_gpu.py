"""Products formed in place with items between a CTA's threads and its largest
item: the same results as the oracle's, and no more time than their outputs
account for."""
import numpy as np
import pytest
import torch

import oracle.rrr

pytestmark = pytest.mark.gpu


def make(size, blk, rng):
    from dtcf_gb300.rrr import Tensor
    t = Tensor("cccc"[:len(size)], size, tuple(s // b for s, b in zip(size, blk)))
    t.tiles.copy_(torch.from_numpy(rng.uniform(-1, 1, t.tiles.numel())).cuda())
    return t


def operands(size, blk):
    rng = np.random.default_rng(sum(size))
    return make((size[0],) * 2, (blk[0],) * 2, rng), make(size, blk, rng), make(size, blk, rng)


@pytest.mark.parametrize("size,blk", [((8, 30, 34, 36), (8, 15, 17, 18)), ((4, 40, 48, 50), (4, 40, 24, 25)),
                                      ((16, 16, 40, 40), (16, 16, 20, 20)), ((13, 33, 30, 50), (13, 11, 15, 25))])
def test_results(size, blk):
    """Items of 384, 512 and (the last of a tile) fewer elements, whole and ragged tiles."""
    from dtcf_gb300.rrr import Contraction
    F, T, C = operands(size, blk)

    def as_oracle(t):
        return dict(tiles=t.tiles.cpu().numpy().reshape(t.num_tiles, -1), addrs=t.addrs, sym=t.sym,
                    block_range=t.block_range, vgrid=t.vgrid)

    want = oracle.rrr.contract(as_oracle(F), as_oracle(T), as_oracle(C), "a,e", "e,b,i,j", "a,b,i,j", 0.5, 1)
    bound = 2.0 ** -53 * (size[0] + 4) * 0.5 * size[0] + 2.0 ** -50 * np.abs(want).max()
    Contraction(F, T, C, mode="fp64", sign=1).contract("a,e", "e,b,i,j", "a,b,i,j", 0.5)
    torch.cuda.synchronize()
    assert np.max(np.abs(C.tiles.cpu().numpy().reshape(want.shape) - want)) <= bound


def test_time_follows_the_outputs():
    """409600 outputs take less than 0.75 of the time of 1048576: they are 0.39 of the work, and 0.95 of it in time
    with every lane of the largest item issuing its products."""
    from dtcf_gb300.rrr import Plan

    def best(size, blk):
        F, T, C = operands(size, blk)
        p = Plan(F, T, C, "a,e", "e,b,i,j", "a,b,i,j", mode="fp64", sign=1)
        out = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            for ev in (a, b):
                ev.record()
                if ev is a:
                    for _ in range(20):
                        p.execute(F, T, C, 0.5)
            torch.cuda.synchronize()
            out.append(a.elapsed_time(b))
        return min(out)

    assert best((16, 16, 40, 40), (16, 16, 20, 20)) < 0.75 * best((16, 16, 64, 64), (16,) * 4)

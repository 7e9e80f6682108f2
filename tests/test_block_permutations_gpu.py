"""Block permutes of any number of permutations: one launch to every sixteen
of them and table of blocks, whatever the blocks' order, bit for bit."""
import itertools
import random

import numpy as np
import pytest
import torch

from launches import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,count,nperm", [
    ((3, 2, 4, 3), 16, 16), ((3, 2, 4, 3), 17, 17), ((3, 2, 4, 3), 4500, 17), ((4, 4, 4, 4), 5000, 24),
    ((4, 4, 4, 4), 30000, 24), ((2, 3, 2, 2, 3, 2), 600, 36), ((2, 1, 2, 3, 2, 2), 8000, 720), ((40, 30, 3, 50), 40, 20),
])
def test_launches_and_bits(widths, count, nperm):
    import dtcf_gb300 as gbx
    rng = random.Random(count + nperm)
    pick = rng.sample(list(itertools.permutations(range(len(widths)))), nperm)
    perms = [pick[b % nperm] for b in range(count)]
    rng.shuffle(perms)
    used = len(set(perms))
    x = torch.rand(count * int(np.prod(widths)), dtype=torch.float64, device="cuda")
    y = torch.full_like(x, np.nan)
    made = launches(lambda st: gbx.transpose_blocks(x, y, perms, widths, stream=st))
    assert len(made) <= -(-used // 16) + count // 4096
    blocks = x.cpu().numpy().reshape((count,) + widths)
    inverse = {p: [p.index(d) for d in range(len(p))] for p in pick}
    want = np.concatenate([b.transpose(inverse[p]).reshape(-1) for b, p in zip(blocks, perms)])
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)

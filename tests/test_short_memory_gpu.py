"""Jobs and residual tables where their branches' regions do not fit but one
region does: they run as a chain, with the same results."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ENOMEM = -2


class budget:
    """What the calling thread's calls may allocate inside the block."""

    def __init__(self, nbytes):
        self.nbytes = int(nbytes)

    def __enter__(self):
        from dtcf_gb300._lib import lib
        assert lib().gbx_alloc_budget(self.nbytes) == 0

    def __exit__(self, *exc):
        from dtcf_gb300._lib import lib
        assert lib().gbx_alloc_budget(-1) == 0


def peak(**kw):
    from dtcf_gb300._lib import lib
    from dtcf_gb300.cc import config
    p = ctypes.c_double()
    assert lib().gbx_cc_footprint(ctypes.byref(config(**kw)), None, ctypes.byref(p), None) == 0
    return p.value


@pytest.mark.parametrize("case", [
    dict(method="ccsd", engine="split", nocc=16, nvir=64, nirrep=1, max_block=16, slices=5, seed=5),
    dict(method="ccsd", engine="fp64", nocc=12, nvir=44, nirrep=1, max_block=11, seed=3),
], ids=lambda c: c["engine"])
def test_job(case):
    from dtcf_gb300 import GbxError
    from dtcf_gb300._lib import lib
    from dtcf_gb300.cc import Job
    chain, side = peak(use_graph=3, **case), peak(use_graph=1, **case)
    assert side > 1.1 * chain
    want = Job(use_graph=0, **case).iterate(3)
    for room, branches in ((2 * side, None), (0.9 * chain + 0.1 * side, 1), (0.3 * chain + 0.7 * side, 1)):
        with budget(room):
            job = Job(use_graph=1, **case)
        assert job.branches() > 1 if branches is None else job.branches() == branches
        if branches == 1:
            assert b"budget" in lib().gbx_last_error()
            assert job.stats().resident_bytes <= room
        assert np.array_equal(job.iterate(3), want)
        job.close()
    with budget(0.4 * chain), pytest.raises(GbxError) as e:
        Job(use_graph=1, **case)
    assert e.value.code == ENOMEM


@pytest.mark.parametrize("mode", ["fp64", "split"])
def test_table(mode):
    from dtcf_gb300 import GbxError, dltc

    def run(prog):
        g = torch.Generator(device="cuda").manual_seed(1)
        written = {x["c"] for x in prog.table["exprs"]}
        for t in range(len(prog.table["tensors"])):
            v = prog.tensor(t)
            v.zero_()
            if t not in written:
                v.copy_(torch.rand(v.numel(), generator=g, device="cuda", dtype=torch.float64) - 0.5)
        prog.run()
        torch.cuda.synchronize()
        return [prog.tensor(t).clone() for t in range(len(prog.table["tensors"]))]

    d = dltc.dims(8, 24, 4, 6)
    prog = dltc.Program("ccd_t2", d, mode=mode)
    assert prog.branches() > 1
    want = run(prog)
    prog.close()
    room, chains = 1 << 30, 0
    while True:
        with budget(room):
            try:
                prog = dltc.Program("ccd_t2", d, mode=mode)
            except GbxError as e:
                assert e.code == ENOMEM
                break
        assert chains == 0 or prog.branches() == 0
        chains += prog.branches() == 0
        assert all(torch.equal(x, y) for x, y in zip(want, run(prog)))
        prog.close()
        room = room * 24 // 25
    assert chains >= 2

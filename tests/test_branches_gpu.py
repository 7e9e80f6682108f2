"""Whether an iteration or a residual table runs as branches: its graph says
so, and a job's memory is what was planned for them."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

JOBS = [
    dict(method="ccd", engine="fp64", nocc=4, nvir=4, nirrep=1, max_block=4, seed=2),
    dict(method="ccsd", engine="fp64", nocc=5, nvir=13, nirrep=1, max_block=3, seed=3),
    dict(method="ccsd", engine="split", nocc=12, nvir=30, nirrep=4, max_block=6, slices=5, seed=4),
    dict(method="ccsd", engine="split", nocc=16, nvir=48, nirrep=1, max_block=16, slices=6, split_all=1, seed=5),
    dict(method="ccd", engine="split", nocc=24, nvir=80, nirrep=2, max_block=20, slices=4, seed=6),
]


@pytest.mark.parametrize("case", JOBS, ids=lambda c: "%s-%s-o%d-v%d" % (c["method"], c["engine"], c["nocc"], c["nvir"]))
def test_jobs(case):
    from dtcf_gb300._lib import lib
    from dtcf_gb300.cc import Job, config
    jobs = {g: Job(use_graph=g, **case) for g in (0, 1, 2, 3)}
    assert jobs[0].branches() == 0
    assert jobs[3].branches() == 1
    assert jobs[1].branches() > 1
    if case["method"] == "ccsd":  # (a CCD program may be one launch after another)
        assert jobs[2].branches() > 1
    for g, job in jobs.items():
        planned = ctypes.c_double()
        assert lib().gbx_cc_footprint(ctypes.byref(config(use_graph=g, **case)), ctypes.byref(planned), None, None) == 0
        if g != 2:  # a program's records come on top of what is planned
            assert abs(job.stats().resident_bytes - planned.value) <= 0.02 * planned.value + (4 << 20)
        job.close()


@pytest.mark.parametrize("mode", ["fp64", "split"])
@pytest.mark.parametrize("which", ["ccd_t2", "ccsd_t1", "ccsd_t2"])
@pytest.mark.parametrize("dims", [(2, 3, 1, 1), (6, 9, 2, 3), (8, 12, 4, 4)])
def test_tables(mode, which, dims):
    from dtcf_gb300 import dltc
    prog = dltc.Program(which, dltc.dims(*dims), mode=mode)
    assert prog.branches() > 1
    prog.close()

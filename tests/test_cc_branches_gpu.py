"""The iteration graph whose independent steps are branches: bit-identical to
the steps issued one by one, repeatedly, for one step and many, beside another
job on another stream and thread, and with the memory that was planned."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [
    dict(method="ccd", engine="fp64", nocc=4, nvir=4, nirrep=1, max_block=4, seed=2),
    dict(method="ccsd", engine="fp64", nocc=5, nvir=13, nirrep=1, max_block=3, seed=3),
    dict(method="ccsd", engine="split", nocc=12, nvir=30, nirrep=4, max_block=6, slices=5, seed=4),
    dict(method="ccsd", engine="split", nocc=16, nvir=48, nirrep=1, max_block=16, slices=6, split_all=1, seed=5),
    dict(method="ccd", engine="split", nocc=24, nvir=80, nirrep=2, max_block=20, slices=4, seed=6),
]


def same(a, b):
    return all(x is None and y is None or np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%s-%s-o%d-v%d" % (c["method"], c["engine"], c["nocc"], c["nvir"]))
def test_same_as_one_by_one(case):
    from dtcf_gb300.cc import Job
    a, b = Job(use_graph=0, **case), Job(use_graph=1, **case)
    st = torch.cuda.Stream()
    assert np.array_equal(a.iterate(1), b.iterate(1))
    with torch.cuda.stream(st):
        eb = b.iterate(6, stream=st)
    assert np.array_equal(a.iterate(6), eb)
    st.synchronize()
    assert same(a.amplitudes(), b.amplitudes())
    # the graph holds the same kernels, in whatever order
    assert b.stats().launches_per_iter > 0


def test_two_jobs_at_once():
    from dtcf_gb300.cc import Job
    alone = [Job(use_graph=1, **c).iterate(5) for c in CASES[1:3]]
    got = [None, None]

    def work(k):
        st = torch.cuda.Stream()
        job = Job(use_graph=1, **CASES[1 + k])
        got[k] = job.iterate(5, stream=st)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(x, y) for x, y in zip(alone, got))

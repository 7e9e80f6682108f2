"""Fused sums cut into items of 256, 512, 1024 and 2048 elements: energies and
amplitudes against the dense oracle, and no more time for the smaller items
than their elements account for."""
import numpy as np
import pytest

from oracle import cc as occ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [1, 2])
@pytest.mark.parametrize("nocc,nvir,max_block", [(8, 24, 7), (10, 30, 30), (10, 30, 11), (10, 40, 10), (11, 41, 9), (12, 48, 24)])
def test_results(nocc, nvir, max_block, graph):
    from dtcf_gb300.cc import Job
    job = Job(method="ccsd", engine="fp64", nocc=nocc, nvir=nvir, nirrep=1, max_block=max_block, seed=4, use_graph=graph)
    ref = occ.CC(occ.System(nocc, nvir, nirrep=1, max_block=max_block, min_block=1, seed=4), "ccsd")
    want = np.array(ref.iterate(3))
    got = np.concatenate([job.energies()[:1], job.iterate(3)])
    assert np.max(np.abs(got - want)) <= 1e-10
    t1, t2 = job.amplitudes()
    assert np.max(np.abs(t2 - ref.t2)) <= 1e-12 and np.max(np.abs(t1 - ref.t1)) <= 1e-12
    job.close()


def test_time_follows_the_elements():
    """The residual's sum at o = 10, v = 40 takes less than 0.9 of the time of o = 16, v = 48: it has 0.27 of the
    elements, and took 1.14 of the time with every slot of the largest item at work."""
    from dtcf_gb300.cc import Job

    def t2_sum(nocc, nvir, max_block):
        job = Job(method="ccsd", engine="split", nocc=nocc, nvir=nvir, nirrep=1, max_block=max_block, seed=1, use_graph=0)
        runs = [[s["ms"] for s in job.profile() if s["kind"] == 1 and s["name"].startswith("t2[")] for _ in range(41)]
        job.close()
        return float(np.median([sum(r) for r in runs[1:]]))

    assert t2_sum(10, 40, 10) < 0.9 * t2_sum(16, 48, 48)

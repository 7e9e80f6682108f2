"""Which jobs of a serving run keep their branches: a job that the budget
cannot hold takes none from the others, and where memory is short the jobs
with the smaller extra workspaces keep theirs."""
import ctypes

import pytest

from dtcf_gb300._lib import lib
from dtcf_gb300.cc import config
from dtcf_gb300.serve import Server

pytestmark = pytest.mark.gpu

LIMIT = 120.0
SMALL = dict(nocc=8, nvir=24, nirrep=1, max_block=8, min_block=1, seed=4, method="ccsd", engine="fp64")
MID = dict(nocc=12, nvir=48, nirrep=1, max_block=12, min_block=1, seed=5, method="ccsd", engine="split")
BIG = dict(nocc=24, nvir=100, nirrep=1, max_block=16, min_block=1, seed=2, method="ccsd", engine="split")


def planned(use_graph, **kw):
    b = ctypes.c_double()
    assert lib().gbx_cc_footprint(ctypes.byref(config(use_graph=use_graph, **kw)), ctypes.byref(b), None, None) == 0
    return b.value


def serve(budget, jobs):
    """jobs: (configuration, arrival times); the run's statistics."""
    s = Server(budget_bytes=budget, slots=2)
    for kw, arrivals in jobs:
        j = s.add_job(config(**kw))
        for t in arrivals:
            s.submit(j, t)
    s.run(LIMIT)
    st = s.stats()
    s.close()
    return st


def test_a_rejected_job_counts_for_nothing():
    side, chain = planned(1, **SMALL), planned(3, **SMALL)
    assert side > 1.1 * chain
    st = serve(1.5 * side, [(SMALL, (0.0, 0.0, 0.1)), (BIG, (0.0,))])
    assert (st["completed"], st["rejected"]) == (3, 1)
    assert st["peak_planned_bytes"] == pytest.approx(side)
    # nor does a job that nothing is asked of
    st = serve(1.5 * side, [(SMALL, (0.0, 0.1)), (MID, ())])
    assert st["peak_planned_bytes"] == pytest.approx(side)


def test_the_smaller_extra_keeps_its_branches():
    small, small_chain, mid, mid_chain = (planned(g, **kw) for kw in (SMALL, MID) for g in (1, 3))
    assert mid - mid_chain > small - small_chain
    budget = mid_chain + small + 0.5 * (mid - mid_chain)
    st = serve(budget, [(SMALL, (0.0, 1.0)), (MID, (0.0, 1.0))])
    assert st["completed"] == 4 and st["evictions"] == 0
    assert st["peak_planned_bytes"] == pytest.approx(mid_chain + small)


def test_a_job_that_fits_as_a_chain_only_is_served():
    side, chain = planned(1, **MID), planned(3, **MID)
    st = serve(0.5 * (side + chain), [(MID, (0.0, 0.0))])
    assert st["completed"] == 2
    assert st["peak_planned_bytes"] == pytest.approx(chain)

"""A running job's next request behind it on the slot's stream: the same
energies in the same order, only while a slot is free, never more than two
deep."""
import numpy as np
import pytest

from dtcf_gb300.cc import Job, config
from dtcf_gb300.serve import Server

pytestmark = pytest.mark.gpu

CASE = dict(nocc=8, nvir=24, nirrep=2, max_block=6, min_block=1, seed=21, method="ccsd", engine="split")
NIT = 24


@pytest.mark.parametrize("slots", [1, 2, 4])
def test_one_job(slots):
    s = Server(budget_bytes=40e9, slots=slots)
    j = s.add_job(config(**CASE))
    for _ in range(NIT):
        s.submit(j, 0.0)
    s.run(120.0)
    rows = sorted(s.results(), key=lambda r: r["iteration"])
    s.close()
    assert [r["iteration"] for r in rows] == list(range(1, NIT + 1)) and all(r["status"] == 0 for r in rows)
    direct = Job(**CASE)
    assert np.array_equal(np.array([r["energy"] for r in rows]), direct.iterate(NIT))
    direct.close()
    start, end = np.array([r["start"] for r in rows]), np.array([r["end"] for r in rows])
    assert np.all(np.diff(start) > 0) and np.all(np.diff(end) >= 0)
    behind = start[1:] < end[:-1]
    assert behind.any() == (slots > 1)
    assert not (start[2:] < end[:-2]).any()


def test_several_jobs_and_the_limit():
    """Requests left when the time limit comes are timed out, those on the GPU finish."""
    s = Server(budget_bytes=40e9, slots=3)
    ids = [s.add_job(config(**dict(CASE, seed=k))) for k in (1, 2)]
    for j in ids:
        for k in range(8):
            s.submit(j, 0.0)
        s.submit(j, 50.0)
    s.run(1.5)
    rows = s.results()
    s.close()
    for j in ids:
        mine = sorted((r for r in rows if r["job"] == j), key=lambda r: r["iteration"])
        assert [r["status"] for r in mine] == [0] * 8 + [-4], mine  # GBX_ETIMEOUT

"""The partial sums of one-call products: no wait for the driver in a call
after a synchronisation, captured and replayed, and from several threads and
streams at once."""
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(16, 16, 5000), (1, 1, 100000), (500, 2, 4000), (3, 2000, 2500), (24, 40, 60000)]


def operands(m, n, k, seed=0):
    rng = np.random.default_rng(m + n + k + seed)
    A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k))
    return A, B, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()


def check(C, A, B, times=1):
    # `times` products added up, any order: each k + 2 roundings of at most the sum of magnitudes
    k = A.shape[1]
    bound = times * 2 * (k + 2) * 2.0 ** -53 * (np.abs(A) @ np.abs(B).T)
    assert np.all(np.abs(C.cpu().numpy() - times * (A @ B.T)) <= times * bound)


def test_no_driver_wait_after_a_synchronisation():
    """256 outputs of 5000 products take less than 60000 of 700, alone: 24 and 104 us; 181 with the default pool."""
    import dtcf_gb300 as gbx

    def alone(m, n, k):
        _, _, a, b = operands(m, n, k)
        c = torch.zeros(m, n, dtype=torch.float64, device="cuda")
        out = []
        for _ in range(40):
            torch.cuda.synchronize()
            t = time.perf_counter()
            gbx.local_contraction(m, n, k, a, b, c, 0, 1, 1.0)
            torch.cuda.synchronize()
            out.append(time.perf_counter() - t)
        return statistics.median(out)

    assert alone(16, 16, 5000) < alone(300, 200, 700)


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_captured_and_replayed(m, n, k):
    import dtcf_gb300 as gbx
    A, B, a, b = operands(m, n, k)
    c = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    gbx.local_contraction(m, n, k, a, b, c, 0, 1, 1.0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        gbx.local_contraction(m, n, k, a, b, c, 0, 1, 1.0, stream=torch.cuda.current_stream())
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    check(c, A, B, 4)


FIRST = """
import numpy as np, torch
import dtcf_gb300 as gbx
rng = np.random.default_rng(1)
A, B = rng.integers(-9, 10, (16, 5000)).astype(float), rng.integers(-9, 10, (16, 5000)).astype(float)
a, b = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
c = torch.zeros(16, 16, dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode="global"):
    gbx.local_contraction(16, 16, 5000, a, b, c, 0, 1, 1.0, stream=torch.cuda.current_stream())
graph.replay()
torch.cuda.synchronize()
assert np.array_equal(c.cpu().numpy(), A @ B.T)
"""


def test_the_first_call_of_a_process_may_be_captured():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", FIRST], check=True, timeout=300, cwd=root)


def test_threads_and_streams():
    import dtcf_gb300 as gbx
    failures = []

    def work(i):
        try:
            st = torch.cuda.Stream()
            data = [operands(*s, seed=i) for s in SHAPES]
            out = [torch.zeros(m, n, dtype=torch.float64, device="cuda") for m, n, _ in SHAPES]
            torch.cuda.synchronize()
            for _ in range(20):
                for (m, n, k), (_, _, a, b), c in zip(SHAPES, data, out):
                    gbx.local_contraction(m, n, k, a, b, c, 0, 1, 1.0, stream=st)
            st.synchronize()
            for (A, B, _, _), c in zip(data, out):
                check(c, A, B, 20)
        except Exception as e:  # noqa: BLE001 (reported by the test's own thread)
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures

"""Groups whose triples take both engines, which run beside one another unless
one touches what the other writes: the sums are right either way, run after
run, in a capture too."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def gpu(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def triple(A, B, C, m, n, k, rs=None, accumulate=0):
    from dtcf_gb300.leaves import Triple
    return Triple(A, B, C, k, 1, k, 1, rs or n, m, n, k, 1.0, accumulate)


def bound(k):
    return 1e-13 * k + 2.0 ** -44 * k  # entries below 1; six slices


@pytest.mark.parametrize("count", [1, 7, 60])
def test_apart(count):
    from dtcf_gb300.leaves import Group, MODE_AUTO
    rng = np.random.default_rng(count)
    ts, keep, want = [], [], []
    for i in range(2 * count):
        m, n, k = (300, 280, 310) if i % 2 else (int(rng.integers(1, 20)), int(rng.integers(1, 20)), int(rng.integers(1, 40)))
        a, b, c = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (m, n))
        d = [gpu(x) for x in (a, b, c)]
        keep.append(d)
        ts.append(triple(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), m, n, k, accumulate=i // 2 % 2))
        want.append((c if i // 2 % 2 else 0) + a @ b.T)
    g = Group(ts, mode=MODE_AUTO)
    assert set(g.info()[0]) == {0, 1}
    start = [d[2].clone() for d in keep]

    def check():
        torch.cuda.synchronize()
        for d, w in zip(keep, want):
            assert np.max(np.abs(d[2].cpu().numpy() - w)) <= bound(d[0].shape[1])

    for run in range(2):
        for d, s in zip(keep, start):
            d[2].copy_(s)
        g.execute()
        check()
    for d, s in zip(keep, start):
        d[2].copy_(s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.execute(stream=torch.cuda.current_stream())
    graph.replay()
    check()


def test_one_reads_what_the_other_writes():
    """A small product lands inside the first operand of a large one: FP64 triples come first."""
    from dtcf_gb300.leaves import Group, MODE_AUTO
    rng = np.random.default_rng(3)
    n = 300
    a, b = rng.uniform(-1, 1, (n, n)), rng.uniform(-1, 1, (n, n))
    x, y = rng.uniform(-0.3, 0.3, (8, 8)), rng.uniform(-0.3, 0.3, (8, 8))
    dA, dB, dX, dY = (gpu(v) for v in (a, b, x, y))
    dC = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    ts = [triple(dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), n, n, n),
          triple(dX.data_ptr(), dY.data_ptr(), dA.data_ptr() + 8 * (17 * n + 5), 8, 8, 8, rs=n)]
    g = Group(ts, mode=MODE_AUTO)
    assert g.info()[0] == [1, 0]
    g.execute()
    torch.cuda.synchronize()
    a[17:25, 5:13] = x @ y.T
    assert np.max(np.abs(dC.cpu().numpy() - a @ b.T)) <= bound(n)

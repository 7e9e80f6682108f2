"""A residual table run as one graph of branches: the same bits as expression
by expression, again and again, on a stream of its own, in a caller's capture
(which takes the kernels themselves), and after a part of the table was run."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def fill(prog, names, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    written = {x["c"] for x in prog.table["exprs"]}
    for t in range(len(names)):
        v = prog.tensor(t)
        v.zero_()
        if t not in written:
            v.copy_(torch.rand(v.numel(), generator=g, device="cuda", dtype=torch.float64) - 0.5)


def snapshot(prog, names):
    torch.cuda.synchronize()
    return [prog.tensor(t).clone() for t in range(len(names))]


def same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("mode", ["fp64", "split"])
@pytest.mark.parametrize("which", ["ccd_t2", "ccsd_t1", "ccsd_t2"])
@pytest.mark.parametrize("dims", [(2, 3, 1, 1), (6, 9, 2, 3), (8, 12, 4, 4)])
def test_same_as_one_by_one(mode, which, dims):
    from dtcf_gb300 import dltc
    prog = dltc.Program(which, dltc.dims(*dims), mode=mode)
    names = prog.table["tensors"]
    n = len(prog.table["exprs"])
    fill(prog, names, 1)
    for i in range(n):
        prog.run(i, 1)
    want = snapshot(prog, names)
    assert any(x.abs().max() > 0 for x in want)
    for _ in range(3):
        fill(prog, names, 1)
        prog.run()
        assert same(want, snapshot(prog, names))
    st = torch.cuda.Stream()
    fill(prog, names, 1)
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        prog.run(stream=st)
    assert same(want, snapshot(prog, names))
    fill(prog, names, 1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        prog.run(stream=torch.cuda.current_stream())
    graph.replay()
    assert same(want, snapshot(prog, names))
    prog.check()

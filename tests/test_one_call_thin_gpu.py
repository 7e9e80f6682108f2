"""One-call products with a side of one or two, or few outputs and long K:
they run on the kernels that planned ones take, in every operand order, at
the shapes where these begin and where K is cut into ranges, and on the tile
kernel just before."""
import numpy as np
import pytest
import torch

from launches import launches

pytestmark = pytest.mark.gpu

ORDERS = [(0, 1), (1, 0), (0, 0), (1, 1)]


def operands(m, n, k, at, bt):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A, B, C = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (m, n))
    dA = torch.from_numpy(np.ascontiguousarray(A.T if at else A)).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B if bt else B.T)).cuda()
    return A, B, C, dA, dB


def call(noalloc, m, n, k, dA, dB, dC, at, bt, alpha, stream):
    from dtcf_gb300._lib import lib
    f = lib().gbx_local_contraction_noalloc if noalloc else lib().gbx_local_contraction
    assert f(m, n, k, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), at, bt, alpha, stream.cuda_stream) == 0


@pytest.mark.parametrize("noalloc", [0, 1])
@pytest.mark.parametrize("at,bt", ORDERS)
@pytest.mark.parametrize("m,n,k,kernel", [
    (400, 1, 400, "gemv"), (399, 1, 400, "tile"), (400, 2, 399, "gemv"), (400, 2, 396, "tile"), (2000, 1, 2000, "gemv"),
    (1, 2000, 2049, "gemv"), (2, 1999, 2500, "gemv"), (5000, 2, 600, "gemv"), (17, 1, 4608, "gemv"), (2, 17, 4607, "tile"),
    (1, 1, 6144, "small_out"), (1, 1, 6143, "tile"), (1, 2, 4096, "small_out"), (16, 16, 4097, "small_out"),
    (20000, 1, 129, "gemv"), (20000, 1, 128, "thin"), (2, 20000, 128, "thin"), (2, 20000, 129, "gemv"),
    (5, 3, 100001, "small_out"), (16, 16, 4095, "tile"), (17, 3, 65, "tile"),
])
def test_kernel_and_result(m, n, k, kernel, at, bt, noalloc):
    A, B, C, dA, dB = operands(m, n, k, at, bt)
    dC = torch.from_numpy(C.copy()).cuda()
    names = launches(lambda st: call(noalloc, m, n, k, dA, dB, dC, at, bt, -0.75, st))
    assert any(kernel in name for name, _ in names), names
    torch.cuda.synchronize()
    # one product, numpy's or the kernel's in any order: k + 2 roundings of at most the sum of magnitudes
    bound = 2 * (k + 2) * 2.0 ** -53 * (0.75 * (np.abs(A) @ np.abs(B).T) + np.abs(C))
    assert np.all(np.abs(dC.cpu().numpy() - (C - 0.75 * (A @ B.T))) <= bound)

"""The dense LU kernels at the sizes where their split changes (GPU tests).

Every element is updated in a fixed order without fused multiply-adds, so the reference below (the
oracle's dense LU; nalgebra's order in numpy) gives equal bits: no tolerance.  Sizes: one column per
CTA and fewer, 32 columns per CTA and one more, the largest systems.  Random values make most
steps swap rows.
"""
import numpy as np
import pytest
import torch

from oracle.oracle_py import linear_solve_csr
from ressim_b200 import ReservoirSimulator, _abi, linear_solve_bsr
from ressim_b200.simulator import dense_solve_noalloc
from test_gpu_direct import seam_system
from test_gpu_parity import _csr_to_bsr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 2, 1), (8, 4, 1), (11, 3, 1), (7, 9, 1), (16, 4, 1), (5, 13, 1), (8, 8, 2), (17, 5, 2)])
def test_direct_lu_equals_oracle_with_row_swaps(dims):
    deck, rhs, ptr, col, val = seam_system(dims)
    n = deck.n_cells
    val = np.random.default_rng(n).standard_normal(len(val))
    x_cpu, rep_cpu = linear_solve_csr(ptr, col, val, rhs, n)
    gpu = ReservoirSimulator.from_deck(deck)
    x_gpu, rep_gpu = linear_solve_bsr(gpu, *_csr_to_bsr(n, ptr, col, val), rhs)
    assert rep_cpu.backend == rep_gpu.backend == _abi.RF_BACKEND_SPARSE_LU
    assert rep_gpu.iterations == rep_cpu.iterations
    assert np.array_equal(x_gpu, x_cpu)


def _inverse(a):
    a, n = a.copy(), len(a)
    perm = np.arange(n)
    for c in range(n):
        p = c + int(np.argmax(np.abs(a[c:, c])))
        a[[c, p]] = a[[p, c]]
        perm[[c, p]] = perm[[p, c]]
        m = a[c + 1:, c] * (1.0 / a[c, c])
        a[c + 1:, c] = m
        a[c + 1:, c + 1:] = -a[c, c + 1:][None, :] * m[:, None] + a[c + 1:, c + 1:]
    x = np.eye(n)[perm]
    for i in range(n - 1):
        x[i + 1:] = -x[i][None, :] * a[i + 1:, i][:, None] + x[i + 1:]
    for i in range(n - 1, -1, -1):
        x[i] = x[i] / a[i, i]
        x[:i] = -x[i][None, :] * a[:i, i][:, None] + x[:i]
    return x


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 200, 256, 257, 299])
def test_dense_inverse_equals_reference_order(n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal((n, n)), rng.standard_normal(n)
    inv, x = _inverse(a), np.zeros(n)
    for c in range(n):
        x = x + inv[:, c] * b[c]
    a_d, b_d = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (a, b))
    x_d = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    dense_solve_noalloc(n, a_d.data_ptr(), b_d.data_ptr(), x_d.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(x_d.cpu().numpy(), x)

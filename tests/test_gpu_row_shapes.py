"""GPU parity at the row lengths, block shapes and widths where the kernels
change how they share a row's work, against the FP64 oracle.

Tolerances: FP64 results differ from the oracle by the order of a row's sum
alone, 1e-12 of sum |a_ij x_j|; with FP32 accumulation a row of at most 5000
terms stays within 5000 * 2^-24 = 3e-4 of it in the worst order and within
1e-5 in the tree and strided orders used (at most 5000 / 32 terms in a chain),
with BF16 values exact after rounding them on the host.
"""
import numpy as np
import pytest

import oracle
import perf_libs_sparse_b200 as pls
from perf_libs_sparse_b200 import workloads as W

pytestmark = pytest.mark.gpu


def csr_of_lengths(lens, n, rng):
    lens = np.minimum(np.asarray(lens, np.int64), n)
    rp = np.zeros(len(lens) + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.choice(n, int(l), replace=False)) for l in lens]).astype(np.int32)
    return rp, col, rng.standard_normal(int(rp[-1]))


def check(y, ref, scale, tol):
    den = np.maximum(np.abs(ref), scale)
    den[den == 0] = 1
    assert (np.abs(np.asarray(y, np.float64) - ref) / den).max() <= tol


# ------------------------------------------------------------------- SELL


@pytest.mark.parametrize("rows", [2_000, 40_000])
@pytest.mark.parametrize("C_,sigma", [(8, 8192), (16, 1024), (32, 4096), (32, 0)])
def test_sell_slices_of_power_law_rows(rows, C_, sigma):
    m, n, rp, c, v = W.zipf_rows(rows, seed=rows)
    x, y0 = W.uniform_vector(n, 2), W.uniform_vector(m, 3)
    A = pls.SpMat.csr(m, n, rp, c, v)
    assert A.force_config(pls.KIND_SELL, C_, sigma, 0) == 0
    assert A.optimize() == 0
    info = A.exec_info()
    if sigma >= 1024:
        assert info["n_split"] > 0
        assert info["n_items"] * C_ <= 2 ** 21  # fits the allocation-free entry point
    ref = oracle.csr_spmv(rp, c, v, x, y=y0, alpha=1.25, beta=-0.5)
    scale = 1.25 * oracle.csr_absdot(rp, c, v, x) + 0.5 * np.abs(y0)
    for _ in range(2):  # the counts of the slices return to zero
        check(A.spmv(x, y0.copy(), alpha=1.25, beta=-0.5), ref, scale, 1e-12)

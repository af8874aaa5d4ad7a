"""CSR products with rows of every length against the batches a lane keeps in flight, grids
of one block up to more rows than one pass of the grid covers, and the CG step's fused inner
product (a solve from each of these sizes).  GPU."""

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
ROWS_ONE_PASS = 148 * 6 * 32


def _dev(a, cuda):
    return torch.as_tensor(np.ascontiguousarray(a), device=cuda)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, ROWS_ONE_PASS, ROWS_ONE_PASS + 17])
def test_product_and_transpose_with_ragged_rows(cuda, n):
    """Each row's sum within len * eps * sum |v x| of the exact sum (a fused multiply-add per
    entry and three additions across the lanes); alpha and beta add two roundings."""
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    rng = np.random.default_rng(n)
    lens = rng.choice([0, 1, 7, 8, 9, 27, 63, 64, 65, 125, 200], size=n)
    indptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    nnz = int(indptr[-1])
    indices = rng.integers(0, n, nnz).astype(np.int32)
    tpos = rng.permutation(nnz).astype(np.int32)
    vals, x = rng.standard_normal(nnz), rng.standard_normal(n)
    y0 = rng.standard_normal(n)
    if n > 33:
        x[n // 2] = np.inf                        # reaches the rows with that column, no other
    d = [_dev(a, cuda) for a in (indptr, indices, tpos, vals, x)]
    row = np.repeat(np.arange(n), lens)
    for trans in (False, True):
        v = vals[tpos] if trans else vals
        with np.errstate(invalid="ignore"):
            prod = v * x[indices]
            clean = np.isfinite(prod)
            hit = np.bincount(row, ~clean, n) > 0
        prod = np.where(clean, prod, 0.0)
        ref = np.bincount(row, prod, n)
        mag = np.bincount(row, np.abs(prod), n)
        for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
            y = _dev(y0, cuda)
            if trans:
                check(lib.hm_csr_spmv_t(n, ptr(d[0]), ptr(d[1]), ptr(d[2]), ptr(d[3]), ptr(d[4]), ptr(y),
                                        alpha, beta, stream_ptr()))
            else:
                check(lib.hm_csr_spmv(n, ptr(d[0]), ptr(d[1]), ptr(d[3]), ptr(d[4]), ptr(y), alpha, beta,
                                      stream_ptr()))
            out = y.cpu().numpy()
            want = alpha * ref + beta * y0
            # the reference itself is a double sum of rounded products: once more the bound
            bound = EPS * (2 * (lens + 4) * abs(alpha) * mag + 4 * np.abs(beta * y0))
            assert np.all(np.abs(out - want)[~hit] <= bound[~hit])
            assert not np.isfinite(out[hit]).any()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, ROWS_ONE_PASS, ROWS_ONE_PASS + 17])
def test_solve_with_the_fused_inner_product(cuda, n):
    """Jacobi-PCG on a strictly dominant matrix: the true residual meets the tolerance (ten
    times it for the recurrence's drift) and a second solve gives the same bits."""
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    rng = np.random.default_rng(n)
    off = rng.uniform(-1.0, 1.0, max(n - 1, 0))
    A = sp.diags([off, np.full(n, 2.5), off], [-1, 0, 1], format="csr") if n > 1 else sp.csr_matrix([[2.5]])
    b = rng.standard_normal(n)
    ip, ix, va, bd, dg = (_dev(a, cuda) for a in (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data,
                                                  b, A.diagonal()))
    work = torch.empty(lib.hm_pcg_workspace_bytes(n) // 8 + 1, dtype=torch.float64, device=cuda)
    out = []
    for _ in range(2):
        x = torch.zeros(n, dtype=torch.float64, device=cuda)
        it, rr = ctypes.c_int(), ctypes.c_double()
        check(lib.hm_pcg(n, ptr(ip), ptr(ix), ptr(va), None, None, 0, None, ptr(dg), ptr(bd), ptr(x), 1e-11,
                         500, 4, ptr(work), ctypes.byref(it), ctypes.byref(rr), stream_ptr()))
        out.append(x.cpu().numpy())
    assert np.linalg.norm(b - A @ out[0]) <= 1e-10 * np.linalg.norm(b)
    assert np.array_equal(out[0], out[1])

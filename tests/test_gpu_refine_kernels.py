"""The refinement's kernels on an analysis that needs no PaStiX library: the matrix-vector
product with 4, 8, 16 and 32 lanes per row, and GMRES over restarts."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from block_structure import bcsc_of, block_structure
from pastix_b200 import native
from test_gpu_wide_panels import analysis

pytestmark = pytest.mark.gpu


# entries per row, rounded up: 3, 5, 7, 9, 21; row counts that leave the last warp ragged
@pytest.mark.parametrize("points,dims,facto", [(7, (67, 1, 1), "potrf"), (7, (11, 13, 1), "getrf"),
                                               (7, (9, 8, 7), "getrf"), (27, (30, 25, 1), "potrf"),
                                               (27, (7, 8, 9), "potrf"), (7, (6, 1, 1), "potrf")])
def test_spmv_lanes(points, dims, facto):
    st, bc, xt, b = analysis(facto, points, dims, 0.01)
    s = native.Solver(st, facto, "fp64")
    s.bcsc_load(bc)
    # a row's error is at most its entries + 2 roundings, each of at most 2^-53 times the
    # sum of |a_ij| |x_j| <= the row sum (|x| <= 1); twice that, since b is rounded too
    vals = np.abs(bc.Uvalues if facto == "getrf" else bc.Lvalues)
    rows = np.add.reduceat(vals, np.asarray(bc.colptr[:-1]))
    tol = 2 * (np.diff(bc.colptr).max() + 2) * 2.0 ** -53 * rows.max()
    for j in range(2):
        assert np.abs(s.spmv(xt[:, j]) - b[:, j]).max() <= tol
    # alpha and beta, two roundings more on terms of twice and three times the size
    y = s.spmv(xt[:, 0], 2.0, -3.0, b[:, 0])
    assert np.abs(y + b[:, 0]).max() <= 6 * tol
    s.close()


@pytest.mark.parametrize("im", [1, 2, 25])
@pytest.mark.parametrize("facto,shift", [("getrf", 0.0), ("sytrf", -0.05)])
def test_gmres_restarts(facto, shift, im):
    st, bc, xt, b = analysis(facto, 7, (17, 16, 15), shift)
    s = native.Solver(st, facto, "fp32")
    s.bcsc_load(bc)
    s.numfact(1e-8)
    x, it, berr = s.refine(b, s.solve(b), "gmres", eps=1e-12, itermax=60, gmres_im=im)
    assert it <= 60 and np.all(np.asarray(berr) <= 1e-12)
    # the reported error is the recurrence's; the true residual adds the roundings of a few
    # products of A x, below 1e-13 of |b| here
    for j in range(2):
        r = np.linalg.norm(b[:, j] - s.spmv(x[:, j])) / np.linalg.norm(b[:, j])
        assert r <= 1.2e-12
    s.close()


def arrowhead(n, dense, facto, full=False):
    """n rows of a diagonal entry (full: of a dense 20 x 20 block) and the dense columns',
    then dense rows of n + 1 entries."""
    st = block_structure([20] * (n // 20) + [dense], [[n // 20]] * (n // 20) + [[]], facto)
    r = np.random.default_rng(4)
    B = sp.csr_matrix(r.uniform(-1, 1, (dense, n)))
    C = B if facto != "getrf" else sp.csr_matrix(r.uniform(-1, 1, (dense, n)))
    D = sp.kron(sp.identity(n // 20), np.full((20, 20), 0.5)) if full else sp.diags([r.uniform(1, 2, n)], [0])
    A = sp.bmat([[D, C.T], [B, sp.diags([np.full(dense, 2.0 * n)], [0])]]).tocsr()
    s = native.Solver(st, facto, "fp64")
    s.bcsc_load(bcsc_of(A, facto))
    return s, A


# 2 to 17 entries in the short rows; n + 1 in the dense ones: below and above 16 steps of 4, 8
# and 16 lanes
@pytest.mark.parametrize("n", [20, 60, 100, 200, 1000])
@pytest.mark.parametrize("dense", [1, 4, 7, 16])
@pytest.mark.parametrize("facto", ["potrf", "getrf"])
def test_spmv_of_an_arrowhead(facto, dense, n):
    s, A = arrowhead(n, dense, facto)
    x = np.random.default_rng(5).uniform(-1, 1, A.shape[0])
    # entries + 2 roundings of at most 2^-53 times the row's sum, on both sides
    tol = 2 * (np.diff(A.indptr) + 2) * 2.0 ** -53 * np.asarray(abs(A).sum(axis=1)).ravel()
    y = s.spmv(x)
    assert np.all(np.abs(y - A @ x) <= tol)
    assert np.all(np.abs(s.spmv(x, 2.0, -3.0, y) + y) <= 6 * tol)
    s.close()


def test_dense_rows_take_whole_warps():
    # a row of 200 000 entries, read by one chain of loads: no longer among rows of 2 entries
    # than among rows of 21, which have a warp each
    def product(full):
        s, A = arrowhead(200000, 1, "potrf", full)
        x = torch.ones(A.shape[0], dtype=torch.float64, device="cuda")
        y = torch.zeros_like(x)
        stream = torch.cuda.Stream()
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(stream):
                a.record()
                s.spmv_device(x.data_ptr(), y.data_ptr(), 1, stream=stream.cuda_stream)
                b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        s.close()
        return min(times)
    assert product(False) <= 1.25 * product(True)

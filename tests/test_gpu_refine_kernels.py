"""The refinement's kernels on an analysis that needs no PaStiX library: the matrix-vector
product with 4, 8, 16 and 32 lanes per row, and GMRES over restarts."""
import numpy as np
import pytest

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

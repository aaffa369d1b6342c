"""Panels of any width on dense matrices (no PaStiX library): the factor's backward error at
the edges of the panel launch's forms -- one to sixteen 64-column steps, the widest row
block that stays resident (384 columns in FP64, 832 in FP32) and the first that does not, the
widest cblk the library takes -- and on ill-conditioned diagonal tiles."""
import numpy as np
import pytest
import scipy.sparse as sp

from block_structure import bcsc_of, dense_structure
from pastix_b200 import native

pytestmark = pytest.mark.gpu

UNIT = {"fp64": 2.0 ** -53, "fp32": 2.0 ** -24}


def dense_factor(st, coef):
    """The coefficients (2D blocks) as one dense matrix, lower blocks."""
    M = np.zeros((st.n, st.n))
    base = 0
    for k in range(st.cblknbr):
        f0, w = st.cblk_fcolnum[k], st.ncols[k]
        for b in range(st.cblk_fblok[k], st.cblk_fblok[k + 1]):
            r0, c = st.blok_frownum[b], base + st.blok_coefind[b]
            h = st.blok_lrownum[b] - r0 + 1
            M[r0:r0 + h, f0:f0 + w] = coef[c:c + h * w].reshape(w, h).T
        base += w * st.cblk_stride[k]
    return M


def spd(n, condition, seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((n, n)))
    A = (q * np.logspace(0, -np.log10(condition), n)) @ q.T
    return (A + A.T) / 2


def dominant(n, facto, seed):
    r = np.random.default_rng(seed)
    A = r.standard_normal((n, n))
    if facto == "sytrf":
        return (A + A.T) / 2 + np.diag(np.where(r.uniform(size=n) < 0.5, -1, 1) * 1.5 * np.sqrt(n))
    return A + np.diag(np.full(n, 1.2 * np.sqrt(n)))


def backward_error(A, widths, facto, prec, solves=None):
    """|A - L U| over |L| |U| (Frobenius) of A rounded to prec; solves: list that receives the
    relative residuals of solutions with 1, 5 and 9 right-hand sides."""
    if prec == "fp32":
        A = A.astype(np.float32).astype(np.float64)
    st = dense_structure(widths, facto)
    s = native.Solver(st, facto, prec)
    s.bcsc_load(bcsc_of(sp.csc_matrix(A), facto))
    s.numfact(1e-20)
    Lc, Uc = s.factor()
    if solves is not None:
        r = np.random.default_rng(7)
        for nrhs in (1, 5, 9):  # the inverses of the diagonal blocks, through each form of the sweeps
            xt = r.uniform(-1, 1, (st.n, nrhs))
            x = s.solve(np.asfortranarray(A @ xt))
            solves.append(np.linalg.norm(A @ (x - xt)) / (np.linalg.norm(A, 2) * np.linalg.norm(xt)))
    s.close()
    M = dense_factor(st, Lc)
    if facto == "potrf":
        L = np.tril(M)
        U = L.T
    else:
        L = np.tril(M, -1) + np.eye(st.n)
        U = np.tril(dense_factor(st, Uc)).T if facto == "getrf" else np.diag(M)[:, None] * L.T
    return np.linalg.norm(A - L @ U) / np.linalg.norm(np.abs(L) @ np.abs(U))


WIDTHS = {"fp64": ([33, 20], [64, 65], [200, 40], [384, 21], [385, 30], [1024, 17]),
          "fp32": ([33, 20], [64, 65], [200, 40], [832, 21], [833, 30], [1024, 17])}


@pytest.mark.parametrize("facto", ["potrf", "sytrf", "getrf"])
@pytest.mark.parametrize("prec,widths", [(p, w) for p in WIDTHS for w in WIDTHS[p]])
def test_widths(facto, prec, widths):
    n = sum(widths)
    A = spd(n, 1e2, 3) if facto == "potrf" else dominant(n, facto, 3)
    # an entry of L U is off by at most n u of its |L| |U|; random roundings of sums cut at 64
    # terms stay near u, wherever the cuts lie
    solves = []
    assert backward_error(A, widths, facto, prec, solves) <= 4 * UNIT[prec]
    # each sweep adds the rounding of its products, with the inverses up to their condition
    # number (10 and less) times that, to the factor's
    assert max(solves) <= 40 * UNIT[prec]


# the same ratio, mean of six matrices, of substitution with sums cut at 32 columns (measured)
CONDITION = {"fp32": 1e5, "fp64": 1e13}
MEAN = {("potrf", "fp32"): {(200, 130): 0.739, (64, 64, 50): 0.682, (60, 40): 0.896, (320, 30): 0.560},
        ("potrf", "fp64"): {(200, 130): 1.012, (64, 64, 50): 1.154, (60, 40): 1.820, (320, 30): 1.226},
        ("sytrf", "fp32"): {(200, 130): 1.229, (64, 64, 50): 1.217, (60, 40): 1.154, (320, 30): 1.156},
        ("sytrf", "fp64"): {(200, 130): 1.242, (64, 64, 50): 1.280, (60, 40): 1.065, (320, 30): 1.222},
        ("getrf", "fp32"): {(200, 130): 0.548, (64, 64, 50): 0.622, (60, 40): 0.677, (320, 30): 0.524},
        ("getrf", "fp64"): {(200, 130): 0.528, (64, 64, 50): 0.665, (60, 40): 0.668, (320, 30): 0.569}}


@pytest.mark.parametrize("facto,prec", MEAN)
def test_rounding(facto, prec):
    # Cholesky on ill-conditioned tiles, whose inverses lose the digits that substitution
    # keeps; LU and LDL^T on dominant ones.  A tenth for another order of the sums
    for widths, bar in MEAN[facto, prec].items():
        n = sum(widths)
        err = [backward_error(spd(n, CONDITION[prec], i) if facto == "potrf" else dominant(n, facto, i), list(widths),
                              facto, prec) for i in range(6)]
        assert np.mean(err) <= 1.1 * bar * UNIT[prec], widths

"""Panels of wide cblks on the GPU against the oracle, on an analysis that needs no PaStiX
library (the geometric nested dissection of perf/cases.py): the row-block launch of LU
(both sides of the factor), Cholesky and LDL^T, with diagonal blocks of
one to five 64-column steps, full and ragged last steps."""
import numpy as np
import pytest

import oracle
from perf import cases as C
from pastix_b200 import native
from pastix_b200.refhost import BCSC

pytestmark = pytest.mark.gpu

# widest cblk: 110 = 64 + 46, 128 = 2 x 64, 200 = 3 x 64 + 8, 306 = 4 x 64 + 50
GRIDS = [(11, 10, 12), (16, 8, 17), (20, 20, 20), (18, 17, 36)]


def analysis(facto, points, dims, shift, device="cuda"):
    case = dict(kind="step", facto=facto, points=points, nx=dims[0], ny=dims[1], nz=dims[2], prec="fp64", nrhs=2,
                shift=shift)
    a = C._analysis(case, device)
    vals, xt, b = C._inputs(case, 3, "cpu")
    v = vals.numpy()
    bc = BCSC(a["st"].n, a["colptr"], a["rowtab"], v[a["lmap"]], v[a["umap"]] if facto == "getrf" else None,
              float(np.linalg.norm(v[a["lmap"]])))
    return a["st"], bc, xt.numpy().T, np.asfortranarray(b.numpy().T)


@pytest.mark.parametrize("dims", GRIDS)
@pytest.mark.parametrize("facto,shift", [("getrf", 0.0), ("potrf", 0.0), ("sytrf", -0.05)])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 2e-4)])
def test_wide_panels_match_oracle(facto, shift, dims, prec, tol):
    # the bars of the parity tests: 1e-12 in FP64; FP32 a few hundred ulps of the
    # factor for the indefinite systems' growth
    st, bc, xt, b = analysis(facto, 7, dims, shift)
    s = native.Solver(st, facto, prec)
    s.bcsc_load(bc)
    piv = s.numfact(1e-8)
    Lg, Ug = s.factor()
    orc = oracle.Oracle(st)
    f = C.FACTO_ID[facto]
    L, U = orc.fillin(bc)
    assert piv == orc.numfact(f, L, U, s.stats()["threshold"]) == 0
    mask = orc.factor_mask(f)
    assert np.linalg.norm((Lg - L)[mask]) <= tol * np.linalg.norm(L[mask])
    if facto == "getrf":
        assert np.linalg.norm(Ug - U) <= tol * np.linalg.norm(U)
    x = s.solve(b)
    s.close()
    if prec == "fp64":
        assert np.linalg.norm(x - xt) <= 1e-11 * np.linalg.norm(xt)


def test_lu_panels_replace_every_small_pivot():
    # a threshold above every pivot: each one is replaced, counted once, and padding is not
    st, bc, _, _ = analysis("getrf", 7, (20, 20, 20), 0.0)
    s = native.Solver(st, "getrf", "fp64")
    s.bcsc_load(bc)
    assert s.numfact(-1e3) == st.n
    s.close()


@pytest.mark.parametrize("facto,shift", [("getrf", 0.0), ("potrf", 0.0), ("sytrf", -0.05)])
def test_forms_without_resident_row_blocks(facto, shift, monkeypatch):
    # the tile-item launch (Cholesky, LDL^T) and the one-CTA LU kernels, which cblks too
    # wide for a resident row block take
    st, bc, xt, b = analysis(facto, 7, (20, 20, 20), shift)
    monkeypatch.setenv("B200_PANEL_TILES", "1")
    s = native.Solver(st, facto, "fp64")
    s.bcsc_load(bc)
    s.numfact(1e-8)
    Lg, Ug = s.factor()
    orc = oracle.Oracle(st)
    L, U = orc.fillin(bc)
    orc.numfact(C.FACTO_ID[facto], L, U, s.stats()["threshold"])
    mask = orc.factor_mask(C.FACTO_ID[facto])
    assert np.linalg.norm((Lg - L)[mask]) <= 1e-12 * np.linalg.norm(L[mask])
    if facto == "getrf":
        assert np.linalg.norm(Ug - U) <= 1e-12 * np.linalg.norm(U)
    x = s.solve(b)
    s.close()
    assert np.linalg.norm(x - xt) <= 1e-11 * np.linalg.norm(xt)

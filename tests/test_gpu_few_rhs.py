"""Sweeps of few right-hand sides through the one-warp leaf kernels (one right-hand side,
up to 4, more than 4) against the oracle's solve, on trees whose narrow cblks have 1 to 32
columns (analysis of perf/cases.py, no PaStiX library needed)."""
import numpy as np
import pytest

import oracle
from perf import cases as C
from pastix_b200 import native
from test_gpu_wide_panels import analysis

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,dims", [(7, (33, 20, 1)), (7, (7, 6, 9)), (7, (13, 12, 11)), (27, (9, 11, 10))])
@pytest.mark.parametrize("facto,shift", [("potrf", 1e-3), ("sytrf", -0.05), ("getrf", 0.0)])
@pytest.mark.parametrize("nrhs", [1, 2, 4, 5])
def test_few_right_hand_sides_match_oracle(points, dims, facto, shift, nrhs):
    if facto == "getrf" and points != 7:
        pytest.skip("the LU matrices are 7-point ones")
    st, bc, _, _ = analysis(facto, points, dims, shift)
    assert st.ncols.min() <= 8 and st.ncols[(st.ncols > 8) & (st.ncols <= 32)].size
    b = np.asfortranarray(np.random.default_rng(nrhs).uniform(-1.0, 1.0, (st.n, nrhs)))
    s = native.Solver(st, facto, "fp64")
    s.bcsc_load(bc)
    s.numfact(1e-8)
    x = s.solve(b)
    orc = oracle.Oracle(st)
    f = C.FACTO_ID[facto]
    L, U = orc.fillin(bc)
    orc.numfact(f, L, U, s.stats()["threshold"])
    s.close()
    xo = orc.solve(f, L, U, b)
    assert np.linalg.norm(x - xo) <= 1e-11 * np.linalg.norm(xo)

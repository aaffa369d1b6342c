"""Chain-shaped trees (a banded matrix in its own order): one cblk per level.  No PaStiX
library."""
import numpy as np
import pytest
import scipy.sparse as sp

from block_structure import bcsc_of, chain_structure
from pastix_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [5, 12, 40])
@pytest.mark.parametrize("facto", ["potrf", "sytrf", "getrf"])
def test_solutions_of_a_chain(facto, width):
    # few and many right-hand sides: the cblks of 12 and 40 columns are all in the dataflow
    # sweeps, those of 5 never are
    n = 60 * width
    st = chain_structure([width] * 60, facto)
    r = np.random.default_rng(2)
    A = sp.diags([r.uniform(-1, 1, n - d) for d in range(1, width + 1)], range(1, width + 1))
    B = A if facto != "getrf" else sp.diags([r.uniform(-1, 1, n - d) for d in range(1, width + 1)],
                                            range(1, width + 1))
    A = (A + B.T + sp.diags(np.full(n, 2.0 * width + 1))).tocsc()  # diagonally dominant
    s = native.Solver(st, facto, "fp64")
    s.bcsc_load(bcsc_of(A, facto))
    assert s.numfact(0.0) == 0
    for nrhs in (1, 7, 8, 33, 64, 66):
        xt = r.uniform(-1, 1, (n, nrhs))
        x = s.solve(np.asfortranarray(A @ xt))
        assert np.linalg.norm(x - xt) <= 1e-13 * np.linalg.norm(xt), nrhs
    s.close()

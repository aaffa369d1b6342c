"""Sweeps of many right-hand sides (row-major vectors, the dataflow launch of the narrow
top of the tree up to 64 of them): every width class of the tiles (16, 32, 48, 64 columns),
odd and ragged numbers, cblks from 1 to 200 columns, against x_true (FP64) and the same
factor's solutions one at a time (FP32).  Analysis of perf/cases.py, no PaStiX library."""
import ctypes
import time

import numpy as np
import pytest
import torch

import oracle
from pastix_b200 import native
from perf import cases as C
from test_gpu_wide_panels import analysis

pytestmark = pytest.mark.gpu

CASES = [("potrf", 7, (20, 20, 20), 0.0), ("sytrf", 7, (13, 12, 17), -0.05), ("getrf", 7, (15, 18, 11), 0.0),
         ("potrf", 27, (9, 23, 10), 1e-3), ("sytrf", 7, (37, 41, 1), -0.01), ("potrf", 7, (7, 1, 1), 0.01)]


def factored(facto, points, dims, shift, prec):
    st, bc, _, _ = analysis(facto, points, dims, shift)
    s = native.Solver(st, facto, prec)
    s.bcsc_load(bc)
    s.numfact(1e-8)
    return st, s


@pytest.mark.parametrize("facto,points,dims,shift", CASES)
def test_fp64_solutions(facto, points, dims, shift):
    st, s = factored(facto, points, dims, shift, "fp64")
    rng = np.random.default_rng(5)
    for nrhs in (8, 9, 16, 17, 31, 34, 48, 50, 64, 65, 130):
        xt = rng.uniform(-1.0, 1.0, (st.n, nrhs))
        x = s.solve(s.spmv(xt))
        err = np.linalg.norm(x - xt, axis=0) / np.linalg.norm(xt, axis=0)
        # rounding times the conditioning of the shifted systems, every column
        assert err.max() <= 1e-10, nrhs
    s.close()


@pytest.mark.parametrize("facto,points,dims,shift", CASES)
def test_fp32_solutions_equal_one_at_a_time(facto, points, dims, shift):
    st, s = factored(facto, points, dims, shift, "fp32")
    b = np.asfortranarray(np.random.default_rng(6).uniform(-1.0, 1.0, (st.n, 67)))
    one = np.stack([s.solve(b[:, j]) for j in range(67)], axis=1)
    for nrhs in (8, 11, 16, 18, 32, 33, 47, 49, 64, 67):
        x = s.solve(b[:, :nrhs])
        d = np.linalg.norm(x - one[:, :nrhs], axis=0) / np.linalg.norm(one[:, :nrhs], axis=0)
        # two summation orders of the same FP32 products: FP32 rounding times the growth
        # of the indefinite systems' solutions
        assert d.max() <= 2e-3, nrhs
        assert np.median(d) <= 1e-4, nrhs
    s.close()


def test_refinement_of_many_right_hand_sides():
    st, s = factored("potrf", 7, (20, 20, 20), 0.0, "tf32x3")
    xt = np.random.default_rng(7).uniform(-1.0, 1.0, (st.n, 21))
    b = s.spmv(xt)
    x, nit, berr = s.refine(b, s.solve(b), "cg")
    s.close()
    assert berr.max() <= 1e-12 and nit <= 3
    assert np.linalg.norm(x - xt) <= 1e-8 * np.linalg.norm(xt)


# cblks of 9 to 32 columns (the 2D grids) and wider ones, of M-matrices and an indefinite system
@pytest.mark.parametrize("facto,points,dims,shift", [("potrf", 7, (20, 20, 20), 0.0), ("potrf", 27, (20, 21, 19), 1e-3),
                                                     ("potrf", 7, (70, 70, 1), 0.0), ("getrf", 7, (22, 20, 21), 0.0),
                                                     ("sytrf", 7, (60, 70, 1), 0.01)])
@pytest.mark.parametrize("low", [-1.0, 0.0])
def test_fp32_many_as_accurate_as_few(facto, points, dims, shift, low):
    # both forms against the 64-bit solve with the same FP32 factor; right-hand sides of one
    # sign give products of one sign, whose rounding must not be one-sided either
    st, s = factored(facto, points, dims, shift, "fp32")
    f = C.FACTO_ID[facto]
    b = np.asfortranarray(np.random.default_rng(8).uniform(low, 1.0, (st.n, 64)))
    exact = oracle.Oracle(st).solve(f, *s.factor(), b)

    def error(nrhs):  # rms over the columns of the relative errors
        x = np.concatenate([s.solve(np.asfortranarray(b[:, i:i + nrhs])).reshape(st.n, -1)
                            for i in range(0, 64 - nrhs + 1, nrhs)], axis=1)
        d = np.linalg.norm(x - exact[:, :x.shape[1]], axis=0) / np.linalg.norm(exact[:, :x.shape[1]], axis=0)
        return np.sqrt((d ** 2).mean())

    few = error(4)
    # the same roundings in another order: a tenth for the sample
    for nrhs in (8, 16, 17, 40, 64):
        assert error(nrhs) <= 1.1 * few, nrhs
    s.close()


def test_withheld_item_ends_the_dataflow_sweep(monkeypatch):
    # the top of the tree in one launch up to 64 columns (fewer launches than level by level,
    # from 65 on); its first item withheld: bounded waits, an error status, and the instance
    # solves again
    st, s = factored("potrf", 7, (20, 20, 20), 0.0, "fp64")
    xt = np.random.default_rng(9).uniform(-1.0, 1.0, (st.n, 66))
    b = s.spmv(xt)
    s.solve(b)
    level_by_level = s.stats()["launches_solve"]
    for nrhs in (8, 17, 33, 64):
        x = s.solve(b[:, :nrhs])
        assert s.stats()["launches_solve"] < level_by_level
        monkeypatch.setenv("B200_TEST_WITHHOLD", "flow")
        t = time.perf_counter()
        with pytest.raises(native.B200Error):
            s.solve(b[:, :nrhs])
        assert time.perf_counter() - t < 20.0
        monkeypatch.delenv("B200_TEST_WITHHOLD")
        assert np.linalg.norm(s.solve(b[:, :nrhs]) - x) <= 1e-13 * np.linalg.norm(x)
    s.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nrhs", [8, 9])
def test_solve_that_allocates_nothing(prec, nrhs):
    st, s = factored("sytrf", 7, (13, 12, 17), 0.05, prec)
    b = np.asfortranarray(np.random.default_rng(10).uniform(-1.0, 1.0, (st.n, nrhs)))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        d = torch.from_numpy(b.T.copy()).cuda()
        assert native.lib().b200_solve_device_noalloc(s.h, nrhs, ctypes.c_void_p(d.data_ptr()), st.n,
                                                      ctypes.c_void_p(stream.cuda_stream)) == 0
    stream.synchronize()
    x = s.solve(b)
    assert np.linalg.norm(d.cpu().numpy().T - x) <= (1e-12 if prec == "fp64" else 1e-5) * np.linalg.norm(x)
    s.close()


@pytest.mark.parametrize("nrhs", [8, 9])
@pytest.mark.parametrize("facto,shift,method", [("potrf", 0.0, "cg"), ("sytrf", -0.05, "gmres")])
def test_refinement_with_an_fp64_factor(facto, shift, method, nrhs):
    # an even number of columns takes the row-major sweeps, an odd one does not
    st, s = factored(facto, 7, (17, 16, 15), shift, "fp64")
    xt = np.random.default_rng(11).uniform(-1.0, 1.0, (st.n, nrhs))
    b = s.spmv(xt)
    x, nit, berr = s.refine(b, np.zeros_like(b), method, eps=1e-13)
    assert berr.max() <= 1e-13 and nit <= 3
    assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)
    s.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_batch_of_systems(prec):
    case = dict(kind="step", facto="sytrf", points=5, nx=16, ny=40, nz=12, prec=prec, nrhs=9, shift=-0.02)
    S = C.prepare(case, 5)
    x = C.run(S)
    torch.cuda.synchronize()
    xt = C.exact(case, 5)
    tol = C.tolerance(case)["rel"]
    assert torch.linalg.norm(x - xt) <= tol * torch.linalg.norm(xt)
    S["s"].close()

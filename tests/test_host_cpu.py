"""The library's host code on a CUDA runtime that computes nothing (fake_cudart.c): what its
entry points do when an allocation fails."""
import glob
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)

PROGRAM = """
import ctypes, sys
sys.path[:0] = [{repo!r}, {here!r}]
import numpy as np
import scipy.sparse as sp
from pastix_b200 import native
native.LIBPATH = {lib!r}
from block_structure import bcsc_of, chain_structure

fake = native.lib()
fake.fake_limit.argtypes = [ctypes.c_size_t]
fake.fake_limit.restype = None
fake.fake_largest.restype = ctypes.c_size_t
fake.fake_nulls.restype = ctypes.c_long


def solver(n, prec):
    st = chain_structure([20] * (n // 20), "potrf")
    s = native.Solver(st, "potrf", prec)
    s.bcsc_load(bcsc_of(sp.diags([np.full(n, 4.0)], [0]).tocsc(), "potrf"))
    s.numfact(0.0)
    return s

"""


@pytest.fixture(scope="session")
def run(tmp_path_factory):
    objs = glob.glob(os.path.join(REPO, "pastix_b200", "lib", "*.o"))
    if not objs:
        pytest.skip("the library's object files are not built")
    d = tmp_path_factory.mktemp("fake")
    subprocess.run(["gcc", "-O1", "-fPIC", "-c", os.path.join(HERE, "fake_cudart.c"), "-o", str(d / "fake.o")], check=True)
    lib = str(d / "libfake.so")
    # -Bsymbolic: the fake's functions, not those of a CUDA runtime that PyTorch has loaded
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", lib, *objs, str(d / "fake.o")], check=True)

    def go(body):
        code = PROGRAM.format(repo=REPO, here=HERE, lib=lib) + body
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return go


def test_scalars_after_a_failed_growth(run):
    # GMRES asks for im + 1 scalars per right-hand side, CG for two: a refused GMRES must not
    # leave the next CG with the capacity of a block that is gone
    run("""
s = solver(20, "fp32")
s.solve(np.ones((20, 100), order="F"))  # a workspace that the refinements fit in
b = np.ones((20, 3), order="F")
s.refine(b, b, "cg")
fake.fake_limit(100)
try:
    s.refine(b, b, "gmres", gmres_im=25)
    raise SystemExit("the allocation was not refused")
except native.B200Error:
    pass
fake.fake_nulls()
s.refine(b, b, "cg")
assert fake.fake_nulls() == 0
""")


def test_creation_is_linear_in_a_chain(run):
    # the schedule of four times the cblks is four times the work (a list built by insertions
    # at its front took sixteen times)
    run("""
import time

def create(ncblk):
    st = chain_structure([12] * ncblk, "potrf")
    t = time.perf_counter()
    s = native.Solver(st, "potrf", "fp64")
    t = time.perf_counter() - t
    s.close()
    return t

create(100)
short, long = (min(create(n) for _ in range(3)) for n in (10000, 40000))
assert long <= 8 * short + 0.02, (short, long)
""")

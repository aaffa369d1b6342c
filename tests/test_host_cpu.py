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


def test_update_records_stay_small(tmp_path):
    # a million of them are filled, uploaded and read for a 512-system forest
    src = tmp_path / "size.cpp"
    src.write_text('#include "b200_internal.h"\nstatic_assert(sizeof(b200::Upd) <= 72, "record");\nint main() {}\n')
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(REPO, "pastix_b200", "csrc"), "-I",
                    "/usr/local/cuda/include", "-fsyntax-only", str(src)], check=True)


def test_row_maps(run):
    # the destination rows of every update, which are uploaded, against a search row by row
    run("""
from block_structure import block_structure, dense_structure
from perf import cases as C

fake.fake_watch.argtypes = [ctypes.c_size_t]
fake.fake_watch.restype = None
fake.fake_watched.restype = ctypes.POINTER(ctypes.c_int)


def expected(st, sides):
    first, last, own, face = st.blok_frownum, st.blok_lrownum, st.cblk_fblok, st.blok_fcblknm
    level = [0] * st.cblknbr
    for k in range(st.cblknbr):
        for f in face[own[k] + 1:own[k + 1]]:
            level[f] = max(level[f], level[k] + 1)
    out = []
    for k in sorted(range(st.cblknbr), key=lambda k: (level[k], k)):
        for j in range(own[k] + 1, own[k + 1]):
            f = face[j]
            row = {}
            at = 0
            for b in range(own[f], own[f + 1]):
                for r in range(first[b], last[b] + 1):
                    row[r] = at
                    at += 1
            for side in range(sides):
                out += [row.get(r, -1) for b in range(j + side, own[k + 1]) for r in range(first[b], last[b] + 1)]
    return out


for facto, st in [("potrf", C._structure(7, 6, 5, 27, "potrf")), ("getrf", C._structure(9, 4, 6, 7, "getrf")),
                  ("potrf", dense_structure([5, 40, 3], "potrf")),
                  # cblk 1 lacks rows that cblk 0 updates it in: entries of -1
                  ("getrf", block_structure([3, 4, 5, 2], [[1, 2, 3], [3], [3], []], "getrf"))]:
    want = expected(st, 2 if facto == "getrf" else 1)
    fake.fake_watch(4 * len(want))
    s = native.Solver(st, facto, "fp64")
    got = fake.fake_watched()
    assert got and got[:len(want)] == want
    s.close()
""")


@pytest.mark.parametrize("nrhs", [8, 9])
def test_solve_without_room_for_padding(run, nrhs):
    # an odd number of FP64 columns is padded to an even one where that fits
    run(f"""
s = solver(2000, "fp64")
fake.fake_limit(2 * 2000 * {nrhs} * 8)
s.solve(np.ones((2000, {nrhs}), order="F"))
""")


def test_trace_runs_the_sweeps_of_the_solve(run):
    # the same launches, one by one: 12-column cblks, whose top of the tree is one launch per
    # sweep row-major and column-major alike, and 60-column ones
    run("""
def counts(s, nrhs):
    s.solve(np.ones((s.n, nrhs), order="F"))
    s.solve_trace(nrhs)
    cls, _ = s.trace_launches()
    return s.stats()["launches_solve"] - 2, int((cls > 0).sum())  # without the permutations

for width in (5, 12, 60):
    st = chain_structure([width] * 40, "potrf")
    s = native.Solver(st, "potrf", "fp64")
    s.bcsc_load(bcsc_of(sp.diags([np.full(st.n, 4.0)], [0]).tocsc(), "potrf"))
    s.numfact(0.0)
    for nrhs in (2, 8, 9, 65):
        solve, trace = counts(s, nrhs)
        assert solve == trace, (width, nrhs, solve, trace)
""")


def test_rule_of_the_row_major_sweeps(run):
    # the sweeps' launches at 7 columns are column-major; FP32 grids on both sides of the line
    run("""
from perf import cases as C

def row_major(dims, facto, prec, nrhs):
    s = native.Solver(C._structure(*dims, 7, facto), facto, prec)
    s.bcsc_load(bcsc_of(sp.diags([np.full(s.n, 4.0)], [0]).tocsc(), facto))
    s.numfact(0.0)
    def launches(k):
        s.solve_trace(k)
        return len(s.trace_launches()[0])
    return launches(nrhs) != launches(7)

for dims, facto, counts in [((9, 9, 9), "potrf", {8: 1, 17: 1}), ((24, 24, 24), "potrf", {8: 1, 17: 1}),
                            ((28, 28, 28), "potrf", {8: 0, 24: 0, 25: 1, 48: 1}),
                            ((32, 32, 32), "getrf", {8: 1, 17: 1}), ((58, 58, 58), "potrf", {8: 0, 33: 0, 48: 1}),
                            ((300, 300, 1), "potrf", {8: 0, 24: 0, 33: 1})]:
    for nrhs, want in counts.items():
        assert row_major(dims, facto, "fp32", nrhs) == bool(want), (dims, nrhs)
    assert row_major(dims, facto, "fp64", 8), dims
""")

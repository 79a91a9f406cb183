"""The expansion's two ways to a station's cell (csrc/fj_cell.h) without a GPU:
locate(), which the plan and the beginning of each chunk of stations use, and
the walk over the cells that the moments kernel takes within a chunk. Where
they differed, a chunk ended in one cell and the next one began in another,
and the moments of a cell were lost."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    return load_rule(tmp_path_factory.mktemp("cell"))


def load_rule(folder):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so = str(folder / "libcell.so")
    # every operation rounded by itself, as the device's intrinsics do
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-march=native", "-shared",
                    "-fPIC", "-I", os.path.join(REPO, "cc-fjpy_b200", "csrc"),
                    os.path.join(REPO, "tests", "cell_rule_check.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    F, I = ctypes.c_float, ctypes.c_int
    lib.cell_disagreements.argtypes = [ctypes.c_longlong, ctypes.c_ulonglong, F]
    lib.cell_disagreements.restype = ctypes.c_longlong
    lib.cell_carries.argtypes = [F, F, F, F, I, ctypes.c_void_p]
    lib.cell_hu.argtypes, lib.cell_hu.restype = [F], ctypes.c_double
    lib.cell_locate.argtypes = [F, F, F, I]
    lib.cell_walk.argtypes = [F, F, F, I, I]
    return lib


# (r, f) whose product's float lies one spacing below a whole number of cells
# that the exact product has reached
@pytest.mark.parametrize("r,f,cell", [(353319.531, 0.96676892, 438), (320676.438, 1.22811925, 505)])
@pytest.mark.parametrize("dy", [0, 1])
def test_carry_over_a_cell_end(rule, r, f, cell, dy):
    cell += 23 * dy  # the halved cells come first
    assert rule.cell_locate(r, f, 500.0, dy) == cell
    assert rule.cell_walk(r, f, 500.0, dy, cell - 2) == cell


@pytest.mark.parametrize("cmin", [500.0, 800.0, 1000.0, 1437.5, 2000.0])
def test_both_ways_end_in_the_same_cell(rule, cmin):
    assert rule.cell_disagreements(20_000_000, int(cmin), cmin) == 0


def test_carries_are_found(rule):
    """The stations that the GPU test puts at chunk ends exist."""
    out = np.zeros(8, dtype=np.float32)
    n = sum(rule.cell_carries(f, 500.0, 2e5, 4e5, 8, out.ctypes.data)
            for f in np.linspace(0.9, 1.1, 64).astype(np.float32))
    assert n > 8

"""Handles of different sizes whose solves run the same resident kernel, from several host threads at once.

A resident solve's shared memory depends on the handle's size; handles are independent, so nothing of one handle's launch
may depend on another's.  Each thread solves on its own handle (tests/cpp/solve_threads.cpp, without the interpreter's
lock between the calls); every result has to be the bits of the same solve alone.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import ssim_gb300 as g
from ssim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def threads(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so, lib_dir = str(tmp_path_factory.mktemp("threads") / "solve_threads.so"), os.path.dirname(_lib.LIB_PATH)
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(HERE, "..", "include"),
                    os.path.join(HERE, "cpp", "solve_threads.cpp"), "-o", so, "-L", lib_dir, "-lssim_gb300",
                    f"-Wl,-rpath,{lib_dir}", "-lpthread"], check=True, capture_output=True, text=True)
    return C.CDLL(so)


def _handle(precision, hexes, blocks):
    X, T = mesh.kuhn_box(hexes, tuple(0.1 * k for k in hexes))
    X = mesh.jitter_interior(X, 0.008, 61)
    fixed = np.where(X[:, 0] == 0.0)[0]
    ts = g.TimeStep(X, T, 1e-2, 1e5, 0.45, 1000.0)
    ts.set_precision(precision)
    ts.set_material(10.0 ** mesh.uniform(62, T.shape[0], 4.0, 6.0), None)
    ts.mark_dirichlet_batched(fixed, np.zeros((fixed.size, 3)))
    ts.set_params(g.default_params(precond=2, pcg_max_blocks=blocks))
    ts.reset("newton")
    ts.update_hessian(False, True, True)
    return ts, np.ascontiguousarray(np.random.default_rng(63).normal(size=X.shape))


@pytest.mark.parametrize("precision,sizes", [
    ("mixed", (((13, 9, 7), 3), ((13, 9, 7), 4))),     # 12 and 9 slices a block, entries on chip
    ("mixed", (((13, 9, 7), 1), ((13, 9, 7), 2))),     # 35 and 18, entries in global memory
    ("fp64", (((10, 10, 10), 0), ((24, 19, 19), 0))),  # one and three slices a block, entries on chip
    ("fp64", (((13, 9, 7), 2), ((13, 9, 7), 3))),      # 18 and 12, entries in global memory
])
def test_handles_of_one_kernel_from_threads(threads, precision, sizes):
    made = [_handle(precision, *s) for s in 2 * sizes]
    n = len(made)
    why = C.create_string_buffer(300)
    bad = threads.solve_threads(n, (C.c_void_p * n)(*[ts._h.value for ts, _ in made]),
                                (C.c_void_p * n)(*[b.ctypes.data for _, b in made]),
                                (C.c_int * n)(*[b.size for _, b in made]), 2000, why, len(why))
    assert bad == 0, (bad, why.value.decode())

"""The FP64 SVD of elem_math.cuh on the host, whose right basis starts in FP32.

A gradient times a power of two has the same U and V and singular values times it, bit for bit, over the range the FP32
start serves (entries from 1e-10 to 1e15): no part of it may leave FP32's range there.  U diag(s) V^T is F to 1e-14 of its
largest entry (some tens of operations of 1.1e-16), U and V are rotations to 1e-14.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def svd(tmp_path_factory):
    from ssim_gb300.build import nvcc

    so = str(tmp_path_factory.mktemp("svd") / "svd.so")
    subprocess.run([nvcc(), "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-o", so,
                    os.path.join(HERE, "host_svd_check.cu")], check=True, capture_output=True)
    lib, dp = C.CDLL(so), C.POINTER(C.c_double)

    def call(F):
        out, F = np.zeros(21), np.ascontiguousarray(F)
        lib.svd64(F.ctypes.data_as(dp), out.ctypes.data_as(dp))
        return out[:9].reshape(3, 3), out[9:12], out[12:].reshape(3, 3)

    return call


@pytest.mark.parametrize("power", [-31, -28, -20, 20, 33, 36, 40, 47])
def test_svd_scales(svd, power):
    rng = np.random.default_rng(81)
    for k in range(200):
        F = rng.uniform(-1, 1, (3, 3))
        if k % 2:  # singular values from 1 down to 1e-3
            F = np.linalg.qr(F)[0] @ np.diag([1.0, 10.0 ** rng.uniform(-2, 0), 10.0 ** rng.uniform(-3, 0)])
        F /= np.abs(F).max()
        U, s, V = svd(F)
        Us, ss, Vs = svd(np.ldexp(F, power))
        assert np.array_equal(U, Us) and np.array_equal(V, Vs) and np.array_equal(np.ldexp(s, power), ss)
        assert np.abs(U * s @ V.T - F).max() <= 1e-14
        for Q in (U, V):
            assert np.abs(Q.T @ Q - np.eye(3)).max() <= 1e-14 and np.linalg.det(Q) > 0

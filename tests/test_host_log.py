"""log(x) and 1/x of the FP64 energy pass (log_rcp.cuh) on the host against numpy's long double, for the arguments the
energy forms (1 + |F|^2 >= 1): the table's interval edges, the neighbourhoods of powers of two, and log-uniform values.
Tolerance: the logarithm is one rounded sum of k ln 2 + log c (two roundings of at most |k| ln 2 + 0.7) and a term below
0.008, so 3e-16 of max(1, log x); the reciprocal is off by r^8 <= 2^-56 and four roundings, 6e-16 of itself."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_log_and_reciprocal(tmp_path):
    from ssim_gb300.build import nvcc

    so = str(tmp_path / "log.so")
    subprocess.run([nvcc(), "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(HERE, "host_log_check.cu")], check=True, capture_output=True)
    rng = np.random.default_rng(0)
    edges = np.array([2.0**k * (1 + j / 64) for k in (0, 1, 2, 3, 10, 60) for j in range(64)])
    x = np.concatenate([edges, np.nextafter(edges[edges > 1], 0), np.nextafter(edges, np.inf), 4 + rng.uniform(-1, 1, 20000),
                        np.exp(rng.uniform(0, 100, 20000)), 1 + 10.0 ** rng.uniform(-15, 0, 20000), [2.0**1022, 1.7e308]])
    l, r = np.zeros_like(x), np.zeros_like(x)
    dp = C.POINTER(C.c_double)
    C.CDLL(so).log_rcp_n(C.c_int(x.size), x.ctypes.data_as(dp), l.ctypes.data_as(dp), r.ctypes.data_as(dp))
    xl = x.astype(np.longdouble)
    assert np.finfo(np.longdouble).eps < 1e-17 or pytest.skip("no long double")
    assert np.all(np.abs(l - np.log(xl)) <= 3e-16 * np.maximum(1, np.log(xl)))
    small = x < 2.0**1000
    assert np.all(np.abs(r[small] * xl[small] - 1) <= 6e-16)
    assert np.all((r[~small] > 0) & (r[~small] < 1e-300))

"""The element stiffness of elem_math.cuh on the host for elongated elements: Kuhn tets of a hex whose longest side is 1 to
1,000 times the others, 10% jitter, in every order of their vertices.

A vertex far from the opposite face has a small shape gradient, and blocks that go with it: every block is compared with
the direct evaluation of test_host_stiffness.py relative to its own two vertices' gradients (mu, lambda |cof F|^2 and
lambda |J - alpha| |F| times |D_v| |D_w|) to that test's tolerances, whose count of operations is that of one block.  The
projected diagonal blocks are positive definite.
"""
import ctypes as C
import itertools

import numpy as np
import pytest

from test_host_stiffness import lib, reference  # noqa: F401 - lib is a fixture


def slivers(ratio, rng):
    corners = np.array(list(itertools.product((0, 1), repeat=3)), float)
    out = []
    for _ in range(3):
        X = corners * [0.05 * ratio, 0.05, 0.05]
        X = X + 0.1 * 0.05 * rng.uniform(-1, 1, X.shape)
        for path in itertools.permutations(range(3)):
            at, ids = np.zeros(3, int), [0]
            for axis in path:
                at[axis] = 1
                ids.append(int(at @ [4, 2, 1]))
            out += [X[list(p)] for p in itertools.permutations(ids)]
    return out


@pytest.mark.parametrize("ratio", [1, 20, 100, 1000])
@pytest.mark.parametrize("name,tol", [("stiffness64", 1e-13), ("stiffness32", 1e-5)])
def test_blocks_of_small_gradients(lib, name, tol, ratio):  # noqa: F811
    rng = np.random.default_rng(ratio)
    S = np.float32 if name == "stiffness32" else np.float64
    fn, dp = getattr(lib, name), C.POINTER(C.c_double)
    for x in slivers(ratio, rng):
        B = np.linalg.inv((x[1:] - x[0]).T).astype(S)
        D = np.concatenate([-(B[0] + B[1] + B[2])[None], B]).astype(float)  # as the kernels form them
        F = (np.eye(3) + 10.0 ** rng.uniform(-4, -0.7) * rng.uniform(-1, 1, (3, 3))).astype(S).astype(float)
        E, nu = 10.0 ** rng.uniform(4, 6), rng.uniform(0.3, 0.48)
        mu, lam = (float(S(m)) for m in (E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))))
        K = np.zeros(144)
        F, D = np.ascontiguousarray(F), np.ascontiguousarray(D)
        fn(F.ctypes.data_as(dp), D.ctypes.data_as(dp), C.c_double(lam), C.c_double(mu), C.c_int(1), C.c_double(1e-4),
           K.ctypes.data_as(dp))
        ref, mag = reference(F, D, lam, mu, True, 1e-4)
        K, n = K.reshape(12, 12), np.sqrt((D * D).sum(1))
        err = np.abs(K - ref).reshape(4, 3, 4, 3).max((1, 3)) / (mag / n.max() ** 2 * np.outer(n, n))
        assert err.max() <= tol, (n, err)
        for v in range(4):
            assert np.linalg.eigvalsh(K[3 * v:3 * v + 3, 3 * v:3 * v + 3])[0] > 0, (v, n)

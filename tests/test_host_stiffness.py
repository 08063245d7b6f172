"""The element stiffness of elem_math.cuh on the host against a direct evaluation: the 9x9 Hessian of the stable
Neo-Hookean energy from its formula, its eigenvalues raised to 1e-3 by numpy's symmetric eigensolver, contracted with
the shape gradients.

Deformation gradients: random strains from 1e-6 to 1, the identity, stretches with two and three equal singular values,
inverted, flat (rank 2), rank 1 and zero elements, and gradients scaled by 1e-3 and 1e3.  Tolerance of the largest entry
of K: 1e-13 in FP64 (a few hundred operations of 1.1e-16, doubled by the projection's sums), 1e-5 in FP32 (the same count
of 6e-8); gradients whose entries are far from 1 make terms of F^4 cancel and are compared relative to the largest of
mu, lambda |cof F|^2 and lambda |J - alpha| |F| times the shape gradients' square.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from ssim_gb300.build import nvcc

    so = str(tmp_path_factory.mktemp("stiff") / "stiff.so")
    subprocess.run([nvcc(), "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-o", so,
                    os.path.join(HERE, "host_stiffness_check.cu")], check=True, capture_output=True)
    return C.CDLL(so)


def cof(F):
    return np.stack([np.cross(F[1], F[2]), np.cross(F[2], F[0]), np.cross(F[0], F[1])])


def reference(F, D, lam, mu, spsd, scale):
    Ic, Cf = (F * F).sum(), cof(F)
    J, alpha = F[0] @ Cf[0], 1 + 0.75 * mu / lam
    f, c = F.reshape(9), Cf.reshape(9)
    H = mu * (1 - 1 / (Ic + 1)) * np.eye(9) + 2 * mu / (Ic + 1) ** 2 * np.outer(f, f) + lam * np.outer(c, c)
    d2 = np.zeros((9, 9))
    for a, b, r in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):  # J = F_r . (F_a x F_b)
        x = F[r]
        K = np.array([[0, x[2], -x[1]], [-x[2], 0, x[0]], [x[1], -x[0], 0]])
        d2[3 * a:3 * a + 3, 3 * b:3 * b + 3] = K
        d2[3 * b:3 * b + 3, 3 * a:3 * a + 3] = K.T
    H = H + lam * (J - alpha) * d2
    if spsd:
        w, Q = np.linalg.eigh(H)
        H = (Q * np.maximum(w, 1e-3)) @ Q.T
    mag = max(mu, lam * (Cf * Cf).sum(), lam * abs(J - alpha) * np.sqrt(Ic), 1e-3) * (D * D).sum(1).max() * scale
    return np.einsum("vj,ijkl,wl->viwk", D, H.reshape(3, 3, 3, 3), D).reshape(12, 12) * scale, mag


def gradients():
    rng = np.random.default_rng(0)
    out = [np.eye(3), np.zeros((3, 3)), np.diag([2.0, 1.0, 1.0]), np.diag([0.5, 0.5, 2.0]), 1.3 * np.eye(3),
           np.diag([1.0, 1.0, -1.0]), np.diag([1.2, 0.9, 0.0]), np.outer([1.0, 2.0, 0.5], [0.3, -1.0, 0.2])]
    for amp in (1e-6, 1e-4, 1e-2, 0.1, 0.3, 1.0):
        out += [np.eye(3) + amp * rng.uniform(-1, 1, (3, 3)) for _ in range(40)]
    out += [rng.normal(size=(3, 3)) * s for s in (1e-3, 1e3) for _ in range(10)]
    for _ in range(20):  # near-equal singular values under rotations
        Q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        R = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        out.append(Q @ np.diag([1.0, 1.0 + 10.0 ** rng.uniform(-12, -3), 1.0 - 10.0 ** rng.uniform(-12, -3)]) @ R.T)
    return out


@pytest.mark.parametrize("name,tol", [("stiffness64", 1e-13), ("stiffness32", 1e-5)])
@pytest.mark.parametrize("spsd", [0, 1])
def test_element_stiffness(lib, name, tol, spsd):
    rng = np.random.default_rng(1)
    fn = getattr(lib, name)
    dp = C.POINTER(C.c_double)
    for F in gradients():
        B = np.linalg.inv(np.eye(3) * 0.05 + 0.01 * rng.uniform(-1, 1, (3, 3)))
        D = np.concatenate([-B.sum(0, keepdims=True), B])
        E, nu = 10.0 ** rng.uniform(4, 6), rng.uniform(0.3, 0.48)
        mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
        if name == "stiffness32":  # the reference sees the same rounded inputs
            F, D, lam, mu = F.astype(np.float32).astype(float), D.astype(np.float32).astype(float), float(np.float32(lam)), float(np.float32(mu))
        K = np.zeros(144)
        F, D = np.ascontiguousarray(F), np.ascontiguousarray(D)
        fn(F.ctypes.data_as(dp), D.ctypes.data_as(dp), C.c_double(lam), C.c_double(mu), C.c_int(spsd), C.c_double(1e-4),
           K.ctypes.data_as(dp))
        ref, mag = reference(F, D, lam, mu, spsd, 1e-4)
        K = K.reshape(12, 12)
        err = np.abs(K - ref).max() / max(np.abs(ref).max(), mag)
        assert np.array_equal(K, K.T) and err <= tol, (F, err)

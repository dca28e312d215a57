"""The FP64 form's element (gbfem_element_fp64.cuh), compiled for the host, against the general element math.

Tolerance: both evaluate the same terms in FP64; the rotation's derivative amplifies roundings by the condition
k of tr(V) I - V (the largest over the smallest sum of two stretches), and a term takes some 200 operations:
200 x 2^-53 x k of the largest entry."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "opensurgsim_gb300", "csrc")


@pytest.fixture(scope="module")
def element(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    lib = str(tmp_path_factory.mktemp("element") / "element_fp64.so")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I" + CSRC, "-o", lib,
                    os.path.join(ROOT, "tests", "support", "element_fp64_host.cu")], check=True, capture_output=True)
    fn = ctypes.CDLL(lib).gbfem_host_element_fp64
    D = ctypes.POINTER(ctypes.c_double)
    fn.argtypes = [D] * 5 + [ctypes.c_double] * 3 + [ctypes.c_int] + [D] * 4
    fn.restype = ctypes.c_int
    return fn


def _rotation(rng, angle):
    a = rng.normal(size=3)
    a /= np.linalg.norm(a)
    K = np.array([[0, -a[2], a[1]], [a[2], 0, -a[0]], [-a[1], a[0], 0]])
    return np.eye(3) + np.sin(angle) * K + (1 - np.cos(angle)) * K @ K


# Rotations over every branch of the quaternion, strains from none to ratios of 1e3, collapsed and turned inside out.
@pytest.mark.parametrize("angle", [0.0, 0.3, 1.5, 2.5, 3.1, np.pi])
@pytest.mark.parametrize("stretch", [(1, 1, 1), (1.01, 0.99, 1), (3, 0.2, 1), (30, 0.03, 1), (1, 0.5, -0.3), (1, 1, 1e-9),
                                     (1, 1, -1), (1e-6, 2e-6, 3e-6), (1e8, 1e8, 2e8)])
@pytest.mark.parametrize("lumped", [0, 1])
def test_same_as_the_general_element(element, angle, stretch, lumped):
    rng = np.random.default_rng(int(10 * angle) + 100 * lumped)
    for _ in range(20):
        x0 = np.vstack([np.zeros(3), np.eye(3)]) * 0.01 + rng.normal(0, 1e-3, (4, 3))
        g = np.linalg.inv(np.vstack([x0.T, np.ones(4)]))[:, :3].copy()
        Q, W = _rotation(rng, angle), _rotation(rng, rng.uniform(0, 3))
        F = Q @ W @ np.diag(stretch) @ W.T
        x = x0 @ F.T + rng.normal(size=3)
        uK, uM = rng.normal(0, 1e-4, (4, 3)), rng.normal(0, 0.1, (4, 3))
        out = [np.zeros(n) for n in (144, 12, 144, 12)]
        ptr = [np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in (x, x0, uK, uM, g)]
        fl = element(*ptr, 0.7, 0.08, 1e-6, lumped, *[a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in out])
        K, rhs, Kgen, rhsGen = out
        assert fl & 7 == fl >> 3
        s = np.sort(np.abs(stretch))[::-1] * np.array([1, 1, np.sign(np.linalg.det(F))])
        cond = (s[0] + s[1]) / max(abs(s[1] + s[2]), 1e-300)
        if cond > 1e7:
            continue  # the factor itself is not defined to FP64
        bound = 200 * 2.0 ** -53 * cond
        low = np.array([4 * a + b for a in range(4) for b in range(a + 1)])
        K, Kgen = K.reshape(16, 9)[low], Kgen.reshape(16, 9)[low]
        assert np.abs(K - Kgen).max() <= bound * np.abs(Kgen).max()
        # Forces cancel from terms of size |K| |x - R x0|.
        size = np.abs(Kgen).max() * (np.abs(x - x[0]).max() + np.abs(x0 - x0[0]).max() + np.abs(uK).max()) + np.abs(uM).max() * 1e-6
        assert np.abs(rhs - rhsGen).max() <= bound * size

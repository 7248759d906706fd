"""The strain decomposition of the device header (csrc/xpbi_math.cuh, strainSVD),
compiled for the host, against NumPy's SVD in 64 bits: every sign of det F,
flattened and inverted particles, and the line between its two branches."""
import ctypes as C
import importlib
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SIGMAS = (1.3, 0.9, 0.72, 0.2, 1e-2, 1e-3, 2e-4, 1e-4, 0.0, -1e-4, -0.1, -0.5, -0.9, -1.0, -1.1)
DIRS = ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 1, 1), (1, -2, 3))


@pytest.fixture(scope="module")
def strain(tmp_path_factory):
    build = importlib.import_module("xpbi-webgpu_gb300.build")
    root = os.path.dirname(HERE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    lib = str(tmp_path_factory.mktemp("strain") / "strain.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I", cuda,
                        "-I", os.path.join(root, "include"), "-I", build.CSRC,
                        os.path.join(HERE, "strain_host.cpp"), "-o", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = C.CDLL(lib).strain_svd

    def run(F, lo=1e-3, hi=1e3):
        H = (np.asarray(F, np.float64) - np.eye(3)).astype(np.float32)
        n = len(H)
        cols = np.ascontiguousarray(np.swapaxes(H, 1, 2))
        out = [np.zeros(s, np.float32) for s in ((n, 3), (n, 3), (n, 3, 3), (n, 3, 3), (n, 3, 3))]
        ptr = [a.ctypes.data_as(C.c_void_p) for a in out]
        fn(cols.ctypes.data_as(C.c_void_p), n, *ptr[:4], C.c_float(lo), C.c_float(hi), ptr[4])
        sig, e, U, V, G = [a.astype(np.float64) for a in out]
        return H.astype(np.float64) + np.eye(3), sig, e, *(np.swapaxes(a, 1, 2) for a in (U, V, G))
    return run


# A column of F V is a sum of at most six rotations' roundings, four operations
# of 6e-8 each: 1.5e-6 of the largest singular value, doubled for the products
# that lead into and out of it.
TOL = 3e-6


def _check(strain, F):
    F, sig, e, U, V, _ = strain(F)
    assert all(np.isfinite(a).all() for a in (sig, e, U, V))
    want = np.linalg.svd(F, compute_uv=False)
    want[:, 2] *= np.where(np.linalg.det(F) < 0, -1.0, 1.0)
    order = np.argsort(-sig, axis=1, kind="stable")
    got = np.take_along_axis(sig, order, 1)
    log = np.take_along_axis(e, order, 1)
    tol = TOL * want[:, :1]
    # a smallest value within rounding of 0 may take either sign: both are clamped
    near = np.abs(want) <= tol
    assert (np.where(near, np.abs(np.abs(got) - np.abs(want)), np.abs(got - want)) <= tol).all()
    lo, hi = np.clip(want - tol, 1e-3, 1e3), np.clip(want + tol, 1e-3, 1e3)
    assert (log >= np.log(lo) - 1e-6).all() and (log <= np.log(hi) + 1e-6).all()
    back = np.einsum("nij,nj,nkj->nik", U, sig, V)
    assert (np.abs(back - F).max(axis=(1, 2)) <= tol[:, 0]).all()
    eye = np.einsum("nji,njk->nik", U, U) - np.eye(3)
    assert np.abs(eye).max() <= 4 * TOL


@pytest.mark.parametrize("axis", DIRS)
def test_one_direction_flattened_or_inverted(strain, axis):
    d = np.array(axis, np.float64) / np.linalg.norm(axis)
    rng = np.random.default_rng(0)
    rot = np.linalg.qr(rng.normal(size=(3, 3)))[0]
    rot *= np.linalg.det(rot)
    F = np.array([np.eye(3) + (s - 1.0) * np.outer(d, d) for s in SIGMAS])
    _check(strain, F)
    _check(strain, np.einsum("ij,njk->nik", rot, F))


@pytest.mark.parametrize("spread", [1e-5, 1e-2, 0.1, 0.2, 0.3, 0.5, 1.0, 3.0])
def test_random_gradients(strain, spread):
    rng = np.random.default_rng(1)
    _check(strain, np.eye(3) + spread * rng.normal(size=(20000, 3, 3)))


def test_reflections_and_nan(strain):
    rng = np.random.default_rng(2)
    q = np.array([np.linalg.qr(m)[0] for m in rng.normal(size=(200, 3, 3))])
    q *= -np.sign(np.linalg.det(q))[:, None, None]  # every one a reflection
    _check(strain, q)
    bad = np.eye(3)[None].copy()
    bad[0, 0, 0] = np.nan
    _, sig, *_ = strain(bad)  # not taken for an undeformed particle
    assert not np.isfinite(sig).all()


@pytest.mark.parametrize("size", [1e-4, 0.05, 0.3, 3.0, 30.0, 300.0])
@pytest.mark.parametrize("hi", [1.001, 1000.0])
def test_clamped_singular_values(strain, size, hi):
    """F with its singular values clamped, as the return maps do: accurate to
    the size of the result, however large F was. (Its rotation feels F's own
    rounding over the smallest sum of two singular values; U and V are off by
    TOL each in at most two columns.)"""
    rng = np.random.default_rng(3)
    F, _, _, _, _, G = strain(np.eye(3) + size * rng.normal(size=(5000, 3, 3)), 0.999, hi)
    u, s, vt = np.linalg.svd(F)
    sign = np.where(np.linalg.det(F) < 0, -1.0, 1.0)
    u[:, :, 2] *= sign[:, None]
    s[:, 2] *= sign
    to = np.clip(s, 0.999, hi)
    want = np.einsum("nij,nj,njk->nik", u, to, vt)
    cond = np.maximum(s[:, 0] / np.maximum(s[:, 1] + s[:, 2], 1e-30), 1.0)
    assert (np.abs(G - want).max(axis=(1, 2)) <= 4 * TOL * to[:, 0] * cond).all()

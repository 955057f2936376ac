"""The correction of eigenvectors with close eigenvalues (opsec_gpu/csrc/polish.h), compiled from the same
header on the CPU: spectra with pairs and groups at every distance, their vectors mixed as an eigensolver
of 48 bits mixes them."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("polish") / "libpolish_check.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                           os.path.join(HERE, "polish_check.cpp")])
    return C.CDLL(so)


def polish(lib, S, X, m):
    k = X.shape[1]
    G, H = np.asfortranarray(X.T @ X), np.asfortranarray(X.T @ S @ X)
    E, lam = np.zeros((k, m), order="F"), np.zeros(m)
    d = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    ok = lib.chk_polish(k, m, d(G), d(H), d(E), d(lam))
    return bool(ok), X[:, :m] + X @ E, lam


def mixed(rng, lam):
    """Vectors of diag(lam), turned among themselves as far as an error of 5e-14 of the largest
    eigenvalue turns them: freely where eigenvalues are closer."""
    n = lam.size
    noise = rng.standard_normal((n, n)) * 5e-14 * lam[0]
    w, X = np.linalg.eigh(np.diag(lam) + 0.5 * (noise + noise.T))
    return X[:, ::-1] + 1e-13 * rng.standard_normal((n, n))  # and not quite orthonormal


GAPS = [0.0, 1e-16, 1e-14, 1e-13, 1e-12, 1e-11, 1e-10, 1e-9, 1e-8, 1e-7, 1e-6]


@pytest.mark.parametrize("group", [2, 3, 6])
@pytest.mark.parametrize("gap", GAPS)
def test_groups_at_every_distance(lib, gap, group):
    rng = np.random.default_rng([group, GAPS.index(gap)])
    n, m = 60, 41  # a group lies across the cut where group divides unevenly
    lam = np.linspace(1.0, 0.05, n // group)[:, None] - gap * rng.uniform(0.5, 1.5, (n // group, group)).cumsum(axis=1)
    lam = -np.sort(-lam.ravel())
    S = np.diag(lam)
    ok, Y, got = polish(lib, S, mixed(rng, lam), m)
    assert ok
    # FP64 of n terms, and half of (1e-6)^2 from pairs of couplings left to first order
    assert np.max(np.abs(Y.T @ Y - np.eye(m))) <= n * EPS + 1e-12
    P = Y.T @ S @ Y
    assert np.max(np.abs(P - np.diag(np.diag(P)))) <= n * EPS
    assert np.max(np.abs(-np.sort(-got) - lam[:m])) <= n * EPS
    assert np.max(np.abs(np.diag(P) - got)) <= n * EPS


def test_chain_of_uneven_distances(lib):
    rng = np.random.default_rng(5)
    lam = np.concatenate([[1.0, 0.9], 0.8 - np.cumsum(10.0 ** rng.uniform(-14, -6, 20)), np.linspace(0.5, 0.1, 30)])
    S = np.diag(lam)
    ok, Y, got = polish(lib, S, mixed(rng, lam), 40)
    assert ok
    assert np.max(np.abs(Y.T @ Y - np.eye(40))) <= lam.size * EPS + 1e-12
    P = Y.T @ S @ Y
    assert np.max(np.abs(P - np.diag(np.diag(P)))) <= lam.size * EPS


def test_refusals(lib):
    rng = np.random.default_rng(6)
    lam = np.concatenate([[1.0], 0.5 + 1e-13 * rng.standard_normal(200)])  # one group of 200
    assert not polish(lib, np.diag(lam), mixed(rng, -np.sort(-lam)), 100)[0]
    lam = np.array([1.0, 0.5, 0.2])
    X = np.eye(3)
    X[0, 1] = np.nan
    assert not polish(lib, np.diag(lam), X, 2)[0]

"""The symmetry check that keeps exactly degenerate surveys with the library's eigensolver
(opsec_gpu/csrc/symmetry.h), compiled from the same header on the CPU, against the spectrum of a matrix
of the cells' separations."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from opsec_gpu import synth

HERE = os.path.dirname(os.path.abspath(__file__))
FULL = 2 * math.pi


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("symmetry") / "libsymmetry_check.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                           os.path.join(HERE, "symmetry_check.cpp")])
    return C.CDLL(so)


def says(lib, sv, cells):
    b, n = (C.c_double * 6)(*sv.bounds), (C.c_int * 3)(*sv.n)
    return bool(lib.chk_forces_degeneracy(sv.coordsys, b, n, C.c_double(sv.L), int(sv.full_sky()), cells.size,
                                          C.c_void_p(cells.ctypes.data)))


def pairs(sv, cells):
    """Neighbouring eigenvalues of sqrt(Nbar_a Nbar_b) exp(-|x_a - x_b| / 60) closer than 1e-12 of the
    largest: FP64 of matrices of at most 216 rows places them within 216 eps ~ 5e-14."""
    x = synth.cell_centres_xyz(sv, cells)
    d = x[:, None] - x[None]
    if sv.L > 0:
        d -= sv.L * np.rint(d / sv.L)
    S = np.sqrt(np.outer(cells["Nbar"], cells["Nbar"])) * np.exp(-np.linalg.norm(d, axis=2) / 60.0)
    ev = np.linalg.eigvalsh(S)
    return int(np.sum(np.diff(ev) < 1e-12 * ev[-1]))


def grid(n, nbar, side=None, L=0.0):
    side = side or [50.0 * k for k in n]
    sv = synth.Survey(synth.COORD_CARTESIAN, (0.0, side[0], 10.0, 10.0 + side[1], -5.0, side[2] - 5.0), n, L=L)
    cells = synth.make_cells(sv, lambda x, y, z: 1.0 + 0 * x, nquad=1)
    u = [(cells[k] + 0.5) / m - 0.5 for k, m in zip(("d1", "d2", "d3"), n)]  # -1/2 .. 1/2
    cells["Nbar"] = nbar(*u)
    return sv, cells


def shell(n, keep, tilt=0.0, phi=(0.0, FULL)):
    sv = synth.Survey(synth.COORD_SPHERICAL, (200.0, 500.0, -0.8, 0.9, phi[0], phi[1]), n)
    cells = synth.make_cells(sv, lambda r, mu, f: 1.0 + 0 * r, nquad=1)
    cells["Nbar"] = 1.0 + 0.3 * cells["d1"] + 0.05 * cells["d2"] ** 2 + tilt * cells["d3"]
    return sv, cells[keep(cells)].copy()


def gauss(x, y, z):
    return np.exp(-2 * (x * x + y * y + z * z))


def swirl(x, y, z):  # a quarter turn in x and y leaves it, a reflection does not
    return gauss(x, y, z) * (1 + 2.0 * x * y * (x * x - y * y)) + 0.1 * z


def roto(x, y, z):  # a quarter turn with z reflected
    return gauss(x, y, z) * (1 + z * (x * x - y * y) + 2.0 * z * x * y)


def third(x, y, z):  # (x, y, z) -> (y, z, x)
    return gauss(x, y, z) * (1 + 0.3 * (x + y + z) + 2.0 * (x * x * y + y * y * z + z * z * x))


def third_reflected(x, y, z):  # (x, y, z) -> (-y, -z, x)
    return third(x, -y, z)


def plain(x, y, z):
    return gauss(x - 0.1, y + 0.05, z) * (1 + 0.2 * x * y + 0.1 * y * z + 0.3 * x)


def everything(c):
    return c["d1"] >= 0


SURVEYS = {
    "cube": (grid((5, 5, 5), gauss), True),
    "quarter turn": (grid((5, 5, 4), swirl), True),
    "quarter turn, other axis": (grid((5, 4, 5), lambda x, y, z: swirl(z, x, y)), True),
    "rotary reflection": (grid((4, 4, 5), roto), True),
    "third": (grid((4, 4, 4), third), True),
    "third, reflected axes": (grid((5, 5, 5), third_reflected), True),
    "square mask": (lambda s: (s[0], s[1][(s[1]["d1"] - 2) ** 2 + (s[1]["d2"] - 2) ** 2 < 8].copy()), True),
    "unequal cells": (grid((5, 5, 4), gauss, side=[250.0, 260.0, 200.0]), False),
    "reflections only": (grid((5, 4, 3), gauss), False),
    "no symmetry": (grid((4, 4, 4), plain), False),
    "periodic, uniform": (grid((4, 5, 6), lambda x, y, z: 1.0 + 0 * x, side=[300.0] * 3, L=300.0), True),
    "periodic in one axis": (grid((3, 6, 4), lambda x, y, z: 1.0 + x + z * z + 0.2 * x * z, side=[300.0] * 3, L=300.0), True),
    "periodic by a third": (grid((3, 6, 4), lambda x, y, z: 1.0 + x + 0.2 * x * z + z * z + 0.3 * np.cos(6 * np.pi * y + 0.3),
                                 side=[300.0] * 3, L=300.0), True),
    "periodic by a half": (grid((3, 6, 4), lambda x, y, z: 1.0 + x + 0.2 * x * z + z * z + 0.3 * np.cos(4 * np.pi * y + 0.3)
                                + 0.1 * x * np.sin(4 * np.pi * y), side=[300.0] * 3, L=300.0), False),
    "uniform, not a whole period": (grid((4, 5, 6), lambda x, y, z: 1.0 + 0 * x, side=[300.0] * 3, L=900.0), False),
    "rings": (shell((3, 4, 7), everything), True),
    "rings left out": (shell((3, 4, 7), lambda c: (c["d2"] != 2) | (c["d1"] != 1)), True),
    "quarter of a turn": (shell((3, 3, 8), lambda c: c["d3"] % 2 == 0), True),
    "half a turn": (shell((3, 3, 6), lambda c: c["d3"] % 3 != 2), False),
    "rings with a gap": (shell((3, 3, 7), lambda c: (c["d3"] != 3) | (c["d1"] != 1)), False),
    "rings, selection in phi": (shell((3, 3, 6), everything, tilt=0.01), False),
    "arcs": (shell((3, 3, 8), everything, phi=(0.0, 3.0)), False),
    "two cells a ring": (shell((4, 5, 2), everything), False),
}


@pytest.mark.parametrize("name", sorted(SURVEYS))
def test_symmetric_surveys_are_the_degenerate_ones(lib, name):
    survey, degenerate = SURVEYS[name]
    sv, cells = survey(grid((5, 5, 4), gauss)) if callable(survey) else survey
    assert (pairs(sv, cells) > 0) == degenerate
    for order in (np.arange(cells.size), np.random.default_rng(3).permutation(cells.size)):
        assert says(lib, sv, cells[order].copy()) == degenerate


def test_exchange_of_axes_alone_also_stays(lib):
    """Reflections force no pairs, but the plain exchange of two axes has always stayed with the library."""
    sv, cells = grid((4, 4, 3), lambda x, y, z: gauss(x, y, z) * (1 + 0.3 * (x + y) + 0.2 * z * x * y))
    assert says(lib, sv, cells) and pairs(sv, cells) == 0

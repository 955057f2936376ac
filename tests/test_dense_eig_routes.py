"""Dense surveys that the engine's own eigensolver leaves to the library: what the statistics say, and
that the library's vectors come back unchanged."""
import numpy as np
import pytest

from opsec_gpu import api, synth

PK = synth.pk_table()


def klt(sv, cells, M, solver):
    with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.1), extra=(f"klt.solver = {solver}",))) as e:
        e.set_pk(*PK)
        ev, B = e.klt(cells, M)
        return ev, B, e.eig_stats()["block"]


def rings_left_out():
    sv, cells = synth.shell_survey(6, 8, 14)
    return sv, cells[cells["d2"] != 0].copy()


@pytest.mark.gpu
def test_statistics_name_the_solver_whose_vectors_came_back():
    """Every (cos, sin) pair of a survey of whole rings is exactly degenerate: the own kernels' check on
    vectors of close eigenvalues may fail there and the library solves.  Its block size says so."""
    sv, cells = rings_left_out()
    auto, lib = klt(sv, cells, 120, "auto"), klt(sv, cells, 120, "dense")
    assert np.array_equal(auto[1], lib[1]) == (auto[2] == 0)
    assert lib[2] == 0


def box(n, nbar, side=None, L=0.0):
    side = side or [50.0 * k for k in n]
    sv = synth.Survey(synth.COORD_CARTESIAN, (0.0, side[0], 0.0, side[1], 0.0, side[2]), n, L=L)
    return sv, synth.make_cells(sv, nbar, nquad=2)


def swirl(x, y, z):  # left alone by a quarter turn about the box's axis, not by a reflection
    x, y = (x - 225.0) / 225.0, (y - 225.0) / 225.0
    return 3e-4 * np.exp(-x * x - y * y - ((z - 180.0) / 300.0) ** 2) * (1 + 0.5 * x * y * (x * x - y * y))


def round_mask():
    sv, cells = box((9, 9, 8), lambda x, y, z: 3e-4 * np.exp(-(((x - 225.0) ** 2 + (y - 225.0) ** 2) / 9e4)) + 0 * z)
    return sv, cells[(cells["d1"] - 4) ** 2 + (cells["d2"] - 4) ** 2 < 26].copy()


def rings_by_mu():
    sv, cells = synth.shell_survey(6, 8, 14)
    return sv, cells[np.lexsort((cells["d3"], cells["d1"], cells["d2"]))].copy()


DEGENERATE = {"swirl": lambda: box((9, 9, 8), swirl), "round mask": round_mask,
              "periodic": lambda: box((8, 9, 10), lambda x, y, z: 3e-4 + 0 * x, [600.0] * 3, 600.0),
              "rings left out": rings_left_out, "rings by mu": rings_by_mu}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(DEGENERATE))
def test_symmetric_surveys_keep_the_library_s_vectors(name):
    sv, cells = DEGENERATE[name]()
    M = cells.size // 5
    auto, lib = klt(sv, cells, M, "auto"), klt(sv, cells, M, "dense")
    np.testing.assert_array_equal(auto[0], lib[0])
    np.testing.assert_array_equal(auto[1], lib[1])
    assert auto[2] == 0

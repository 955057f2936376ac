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

"""The dense eigensolve of open boxes on the engine's own kernels: the ends of its range, the
orders where its kernels change shape, and what stays with the library."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


def box(n, tilted=True):
    side = [50.0 * k for k in n]
    sv = synth.Survey(synth.COORD_CARTESIAN, (0.0, side[0], 0.0, side[1], 0.0, side[2]), n)

    def sel(x, y, z):
        t = (0.42, 0.57, 0.5) if tilted else (0.5, 0.5, 0.5)
        q = sum(w * (v / s - c) ** 2 for v, s, c, w in zip((x, y, z), side, t, (1.0, 1.3, 0.8) if tilted else (1, 1, 1)))
        return 3e-4 * np.exp(-4.0 * q)

    return sv, synth.make_cells(sv, sel, nquad=2)


def klt(sv, cells, M, solver):
    k, P = synth.pk_table()
    with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.1), extra=(f"klt.solver = {solver}",))) as e:
        e.set_pk(k, P)
        ev, B = e.klt(cells, M)
        return ev, B, e.signal_block(cells), e.eig_stats()["block"]


@pytest.mark.parametrize("n", [(8, 8, 8), (3, 19, 9), (4, 16, 16), (5, 11, 19), (8, 16, 16), (3, 29, 24), (16, 16, 16)])
def test_eigenpairs_match_the_library(n):
    sv, cells = box(n)
    M = cells.size // 5
    ev, B, S, block = klt(sv, cells, M, "auto")
    lib = klt(sv, cells, M, "dense")[0]
    assert block >= M  # the own kernels ran (candidates solved for)
    lam0 = lib[0]
    # FP64 of 4,096 terms: 4096 eps ~ 9e-13 of the largest, an order of margin for the residual
    assert np.max(np.abs(ev - lib)) <= 1e-12 * lam0
    assert np.max(np.abs(B @ S - ev[:, None] * B)) <= 1e-11 * lam0
    assert np.max(np.abs(B @ B.T - np.eye(M))) <= 1e-11


@pytest.mark.parametrize("n,tilted", [((7, 7, 7), True), ((8, 8, 8), False), ((9, 8, 8), False)])
def test_small_and_degenerate_problems_stay_with_the_library(n, tilted):
    sv, cells = box(n, tilted)
    M = cells.size // 5
    auto, dense = klt(sv, cells, M, "auto"), klt(sv, cells, M, "dense")
    np.testing.assert_array_equal(auto[0], dense[0])
    np.testing.assert_array_equal(auto[1], dense[1])

"""The dense eigensolve of boxes that a symmetry almost leaves alone: pairs of eigenvalues at distances from
1e-6 of the largest down to where the symmetry check takes them for equal."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("n", [(6, 6, 18), (12, 12, 10)])
@pytest.mark.parametrize("tilt", [1e-5, 1e-6, 1e-7, 1e-8, 3e-9, 1.2e-9])
def test_close_pairs(n, tilt):
    side = [50.0 * k for k in n]
    sv = synth.Survey(synth.COORD_CARTESIAN, (0.0, side[0], 0.0, side[1], 0.0, side[2]), n)
    cells = synth.make_cells(sv, lambda x, y, z: 3e-4 * (1 + tilt * (x - 2 * y) / side[0]) * np.exp(
        -4.0 * sum((v / s - 0.5) ** 2 for v, s in zip((x, y, z), side))), nquad=2)
    N, M = cells.size, cells.size // 5
    out = {}
    for solver in ("auto", "dense"):
        with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.1), extra=(f"klt.solver = {solver}",))) as e:
            e.set_pk(*synth.pk_table())
            out[solver] = e.klt(cells, M)
            if solver == "auto":
                assert e.eig_stats()["block"] >= M  # not the library
                S = e.signal_block(cells)
    ev, B = out["auto"]
    lam0 = out["dense"][0][0]
    assert np.min(-np.diff(out["dense"][0])) < 1e-6 * lam0
    # FP64 sums of N terms; vectors of two couplings to first order 1e-13 more
    assert np.max(np.abs(ev - out["dense"][0])) <= N * EPS * lam0
    assert np.max(np.abs(B @ B.T - np.eye(M))) <= N * EPS + 1e-13
    P = B @ S @ B.T
    i, j = np.nonzero(np.abs(ev[:, None] - ev[None]) < 1e-6 * lam0)
    assert np.max(np.abs(P - np.diag(np.diag(P)))[i, j]) <= N * EPS * lam0

"""The last stages at the edges of their kernels' splits: pixel values of a build against the dense dot
product, and the epilogue over numbers of bands, pivots off the diagonal included."""
import numpy as np
import pytest

import oracle as O
from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 4), (1, 4, 33), (5, 3, 31), (3, 2, 64), (1, 2, 300), (3, 1, 130)])
def test_pixel_values_of_a_build(dims):
    sv, cells = synth.shell_survey(*dims)
    bands = synth.band_edges(2, 0.0, 0.2)
    M = max(2, min(40, cells.size // 3))
    counts = synth.grf_counts(sv, cells)
    with api.Engine(api.make_config(sv, bands=bands)) as e:
        e.set_pk(*synth.pk_table())
        r = e.fisher_build(cells, counts, M, mixing="identity")
        ev, B = e.klt(cells, M)
        y = e.dot(cells, counts, B)
        g = e.estimate(ev, e.comma(cells, B), y, "identity")
    # FP32 projections of the same modes by two routes: each term 1e-5 off the larger of q and f at most
    q, ref = r["q"] + r["f"], g["q"] + g["f"]
    assert np.max(np.abs(q - ref)) <= 1e-5 * np.max(np.abs(ref) + np.abs(g["f"]))


@pytest.mark.parametrize("nb", [1, 2, 15, 16, 31, 32, 33, 64, 70])
def test_epilogue_over_bands(nb):
    rng = np.random.default_rng(nb)
    M = 60
    sv, cells = synth.shell_survey(2, 2, 4)
    bands = synth.band_edges(nb, 0.0, 0.4)
    evals = np.sort(rng.uniform(0.05, 4.0, M))[::-1]
    # neighbouring bands share a part of their sign-alternating matrices: pivots leave the diagonal
    A = rng.standard_normal((nb, M, M))
    A = A + np.transpose(A, (0, 2, 1))
    A[1:] += 3.0 * A[:-1]
    Dp = np.stack([O.pack_upper(a) for a in A])
    y = rng.standard_normal(M)
    with api.Engine(api.make_config(sv, bands=bands)) as e:
        e.set_pk(*synth.pk_table())
        got = e.estimate(evals, Dp, y, "inverse")
    F = got["F"]
    ref = O.estimate_epilogue(F, got["q"] + got["f"], got["f"], "inverse")
    tol = 64 * nb * np.finfo(float).eps * np.linalg.cond(F)
    for k in ("M", "W", "phat"):
        assert np.max(np.abs(got[k] - ref[k])) <= tol * np.max(np.abs(ref[k])), k

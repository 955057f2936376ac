"""The block eigensolver at the edges of its range: block orders around its chunk (64 columns),
warp and cluster splits, the smallest and largest orders, one to many blocks."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


# (nr, nmu, nphi): odd nmu keeps one block of nr nmu per azimuthal order, even nmu two of half that.
# The first four are small surveys, which keep their own kernels.
@pytest.mark.parametrize("dims", [(1, 3, 6), (4, 1, 5), (13, 5, 9), (40, 5, 40), (1, 6, 172), (2, 4, 130), (1, 10, 103),
                                  (4, 6, 128), (9, 14, 9), (8, 16, 8), (13, 10, 8), (19, 10, 6), (32, 6, 6), (97, 2, 6),
                                  (43, 6, 5), (37, 14, 4), (27, 38, 4), (31, 66, 4), (91, 11, 9)])
def test_eigenpairs_of_every_block_shape(dims):
    sv, cells = synth.shell_survey(*dims)
    k, P = synth.pk_table()
    M = max(1, cells.size // 3)
    out = {}
    for eig in ("own", "batched"):
        with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.2), extra=[f"azimuthal.eig = {eig}"])) as e:
            e.set_pk(k, P)
            out[eig] = e.klt(cells, M)
            if eig == "own":
                assert e.eig_stats()["iterations"] == 1  # not the library's fallback
                S = e.signal_block(cells)
    ev, B = out["own"]
    lam0 = out["batched"][0][0]
    # double-FP32 keeps 47 bits: 7e-15 a step, at most 1023 steps
    assert np.max(np.abs(ev - out["batched"][0])) <= 1e-11 * lam0
    assert np.max(np.abs(B @ S - ev[:, None] * B)) <= 1e-11 * lam0
    # vectors of eigenvalues 1e-6 of the block scale apart, each good to 1e-14 of it
    assert np.max(np.abs(B @ B.T - np.eye(M))) <= 2e-8

"""Vectors of nearly equal eigenvalues of one block: an odd number of mu cells leaves the modes even and odd
in mu together, many of them in pairs."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(20, 33, 14), (13, 45, 15), (37, 15, 18), (16, 27, 20)])
def test_vectors_of_close_pairs_are_orthogonal(dims):
    sv, cells = synth.shell_survey(*dims)
    M = cells.size // 5
    with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.1), extra=("azimuthal.eig = own",))) as e:
        e.set_pk(*synth.pk_table())
        _, B = e.klt(cells, M)
        assert e.eig_stats()["iterations"] == 1
    # vectors of eigenvalues closer than 1e-6 of the block's scale are orthogonalised; beyond, each is off by
    # its shift's error over the distance: two units in the last place of an eigenvalue of that scale,
    # 4.4e-16 / 1e-6, of each of the two
    assert np.max(np.abs(B @ B.T - np.eye(M))) <= 9e-10

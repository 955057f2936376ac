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


@pytest.mark.parametrize("dims,thickness,part", [((37, 15, 16), 60.0, 1), ((37, 15, 16), 20.0, 4), ((20, 31, 14), 100.0, 1),
                                                 ((20, 32, 14), 20.0, 1)])
def test_thin_shells(dims, thickness, part):
    """Shells far thinner than the correlation length: most eigenvalues of a block are close to others."""
    sv, cells = synth.shell_survey(*dims, rmin=200.0, rmax=200.0 + thickness, rc=200.0 + thickness / 2, width=thickness / 2)
    M = cells.size // part
    ev = {}
    for eig in ("own", "batched"):
        with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.1), extra=(f"azimuthal.eig = {eig}",))) as e:
            e.set_pk(*synth.pk_table())
            ev[eig], B = e.klt(cells, M)
            if eig == "own":
                assert e.eig_stats()["iterations"] == 1
                S, own = e.signal_block(cells), B
    lam0 = ev["batched"][0]
    # as the block eigensolver's other tests; orthogonality as above
    assert np.max(np.abs(ev["own"] - ev["batched"])) <= 1e-11 * lam0
    assert np.max(np.abs(own @ S - ev["own"][:, None] * own)) <= 1e-11 * lam0
    assert np.max(np.abs(own @ own.T - np.eye(M))) <= 9e-10

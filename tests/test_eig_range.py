"""The own eigensolvers over FP64's range of S and of its rows: surveys scaled as a whole, and with cells
far in the tail of the selection, first rows and last ones."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu

PK = synth.pk_table()


def klt(sv, cells, M, extra):
    with api.Engine(api.make_config(sv, bands=synth.band_edges(2, 0.0, 0.1), extra=(extra,))) as e:
        e.set_pk(*PK)
        ev, B = e.klt(cells, M)
        return ev, B, e.signal_block(cells), e.eig_stats()


# all cells times a factor, or the cells picked by a slice times one
CHANGES = {"x1e-16": (slice(None), 1e-16), "x1e-36": (slice(None), 1e-36), "x1e25": (slice(None), 1e25),
           "first arc 1e-33": ("first", 1e-33), "first arc 1e-60": ("first", 1e-60), "inner arc 1e-33": ("inner", 1e-33)}


# a small survey's kernels, a cluster of one CTA, odd N_mu on clusters of several
@pytest.mark.parametrize("dims", [(6, 6, 9), (8, 16, 16), (37, 15, 18)])
@pytest.mark.parametrize("change", sorted(CHANGES))
def test_blocks(dims, change):
    sv, cells = synth.shell_survey(*dims)
    which, factor = CHANGES[change]
    if which == "first" or which == "inner":  # an arc and its mirror image in mu
        i, j = (0, 0) if which == "first" else (dims[0] // 2, dims[1] // 2 - 1)
        which = (cells["d1"] == i) & ((cells["d2"] == j) | (cells["d2"] == dims[1] - 1 - j))
    cells["Nbar"][which] *= factor
    M = cells.size // 5
    ev, B, S, stats = klt(sv, cells, M, "azimuthal.eig = own")
    lib = klt(sv, cells, M, "azimuthal.eig = batched")[0]
    assert stats["iterations"] == 1 and stats["block"] >= M // 2
    lam0 = lib[0]
    # the bounds of the block eigensolver's other tests: double-FP32 keeps 47 bits, 7e-15 a step
    assert np.max(np.abs(ev - lib)) <= 1e-11 * lam0
    assert np.max(np.abs(B @ S - ev[:, None] * B)) <= 1e-11 * lam0
    assert np.max(np.abs(B @ B.T - np.eye(M))) <= 2e-8


DENSE = {"x1e-16": (slice(None), 1e-16), "x1e-36": (slice(None), 1e-36), "x1e25": (slice(None), 1e25),
         "first cell 1e-30": (slice(0, 1), 1e-30), "first cell 1e-60": (slice(0, 1), 1e-60),
         "last cell 1e-33": (slice(-1, None), 1e-33), "100 cells 1e-33": (slice(0, 100), 1e-33),
         "fading": (slice(0, 300), 10.0 ** -np.linspace(0, 45, 300))}


@pytest.mark.parametrize("change", sorted(DENSE))
def test_dense(change):
    n = (8, 8, 8)
    sv = synth.Survey(synth.COORD_CARTESIAN, (0.0, 400.0) * 3, n)
    cells = synth.make_cells(sv, lambda x, y, z: 3e-4 * np.exp(
        -4 * ((x / 400 - 0.42) ** 2 + 1.3 * (y / 400 - 0.57) ** 2 + 0.8 * (z / 400 - 0.5) ** 2)), nquad=2)
    which, factor = DENSE[change]
    cells["Nbar"][which] *= factor
    M = 100
    ev, B, S, stats = klt(sv, cells, M, "klt.solver = auto")
    lib = klt(sv, cells, M, "klt.solver = dense")[0]
    assert stats["block"] >= M
    lam0 = lib[0]
    # as tests/test_dense_eig_sizes.py
    assert np.max(np.abs(ev - lib)) <= 1e-12 * lam0
    assert np.max(np.abs(B @ S - ev[:, None] * B)) <= 1e-11 * lam0
    assert np.max(np.abs(B @ B.T - np.eye(M))) <= 1e-11

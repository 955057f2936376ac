"""Bands that share the launches of the tensor-core projection."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,M", [(1, 300), (5, 40), (13, 2000), (21, 300)])
def test_bands_that_share_launches(nb, M):
    """Bands go through the tensor-core kernels several a launch: one, all, and two launches of unequal
    numbers (13 bands of 2,000 modes), against the plain FP32 kernels band by band."""
    sv, cells = synth.box_survey(13)
    cells = cells[:2100]
    modes = np.linalg.qr(np.random.default_rng(M).standard_normal((cells.size, M)))[0].T
    got = {}
    for proj in ("tc", "simt"):
        with api.Engine(api.make_config(sv, bands=synth.band_edges(nb, 0.0, 0.4), extra=[f"projection = {proj}"])) as e:
            e.set_pk(*synth.pk_table())
            got[proj] = e.comma(cells, modes)
    for p in range(nb):
        assert np.max(np.abs(got["tc"][p] - got["simt"][p])) <= 1e-5 * np.max(np.abs(got["simt"][p])), p


@pytest.mark.parametrize("dims,nb", [((2, 2, 8), 1), ((8, 16, 8), 37), ((8, 16, 8), 41), ((7, 5, 12), 41), ((16, 16, 10), 11)])
def test_band_blocks_that_share_launches(dims, nb):
    """The FP32 band blocks go several bands a launch (38 at 64 arcs a block): all in one, a last launch of
    few, against the FP64 blocks, which go one by one."""
    sv, cells = synth.shell_survey(*dims)
    counts = synth.grf_counts(sv, cells)
    M = cells.size // 4
    F = {}
    for gemm in ("tc", "f64"):
        with api.Engine(api.make_config(sv, bands=synth.band_edges(nb, 0.0, 0.4), extra=[f"azimuthal.gemm = {gemm}"])) as e:
            e.set_pk(*synth.pk_table())
            F[gemm] = e.fisher_build(cells, counts, M, mixing="identity")["F"]
    # FP32 blocks and products against FP64 ones: 1e-6 of the largest element, as the projection's other tests
    assert np.max(np.abs(F["tc"] - F["f64"])) <= 2e-6 * np.max(np.abs(F["f64"]))

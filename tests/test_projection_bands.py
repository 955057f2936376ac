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

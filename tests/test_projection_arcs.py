"""The tensor-core projection on grids whose arcs have 16, 32 or 64 cells, on part of the sky and on
all of it, against the CUDA-core projection of the same modes."""
import math

import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi,full", [(16, False), (16, True), (32, False), (64, False), (64, True), (15, False)])
def test_tensor_core_projection_matches_cuda_cores(nphi, full):
    bounds = (200.0, 1000.0, -0.5, 0.8, 0.0, 2 * math.pi) if full else (200.0, 1000.0, -0.5, 0.8, 0.3, 2.0)
    sv = synth.Survey(synth.COORD_SPHERICAL, bounds, (4, 5, nphi))
    cells = synth.make_cells(sv, lambda r, mu, phi: 3e-4 * np.exp(-(((r - 600.0) / 250.0) ** 2)) * (1 + 0.2 * mu),
                             nquad=3)
    modes = np.ascontiguousarray(np.linalg.qr(np.random.default_rng(4).standard_normal((cells.size, 37)))[0].T)
    k, P = synth.pk_table()
    out = {}
    for proj in ("tc", "simt"):
        with api.Engine(api.make_config(sv, bands=synth.band_edges(3, 0.0, 0.09), extra=(f"projection = {proj}",))) as e:
            e.set_pk(k, P)
            out[proj] = e.comma(cells, modes)
    # FP16 hi/lo operands carry 22 bits and the accumulator truncates: 1e-5 of the largest C_p, as
    # the projection's other tests
    assert np.max(np.abs(out["tc"] - out["simt"])) <= 1e-5 * np.max(np.abs(out["simt"]))

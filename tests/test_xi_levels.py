"""The xi tables over every way a group of r is summed: few and many blocks of moments, table
nodes one by one (table 0 at large r, very wide bands), r = 0, group remainders."""
import numpy as np
import pytest

import oracle as O
from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu

NARROW = [(0.0, 0.01), (0.01, 0.02), (0.39, 0.4)]
WIDE = [(0.0, 0.3), (0.2, 2.7), (0.0, 9.0)]


@pytest.mark.parametrize("layout,bands", [((256, 4096, 10.0, 20000.0), NARROW), ((512, 256, 200.0, 20000.0), WIDE),
                                          ((33, 95, 7.5, 3100.0), NARROW + WIDE), ((7, 12, 900.0, 60000.0), WIDE)])
def test_xi_tables_match_the_term_by_term_sums(layout, bands):
    k, P = synth.pk_table()
    sv, _ = synth.shell_survey(3, 4, 8)
    with api.Engine(api.make_config(sv, bands=bands, layout=layout)) as e:
        e.set_pk(k, P)
        r, xi = e.xi_tables()
    ref = O.xi_tables(k, P, bands, layout)
    scale = np.maximum(np.max(np.abs(ref), axis=1, keepdims=True), 1e-300)
    # 1e-12 of max |xi| per table, as the tables' parity test
    assert np.max(np.abs(xi - ref) / scale) <= 1e-12

"""The xi table of a P(k) in other units, over FP64's range of them."""
import numpy as np
import pytest

import oracle as O
from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-300, -100, -60, 60, 95, 105, 300])
@pytest.mark.parametrize("layout", [(256, 4096, 10.0, 20000.0), (512, 256, 200.0, 20000.0)])
def test_xi_follows_the_units_of_the_power_spectrum(layout, power):
    k, P = synth.pk_table()
    bands = synth.band_edges(2, 0.0, 0.1)
    sv, _ = synth.shell_survey(3, 4, 8)
    with api.Engine(api.make_config(sv, bands=bands, layout=layout)) as e:
        e.set_pk(k, P)
        one = e.xi_tables()[1]
        e.set_pk(k, P * 2.0 ** power)
        xi = e.xi_tables()[1]
    np.testing.assert_array_equal(xi[0], one[0] * 2.0 ** power)  # a power of two moves no rounding
    np.testing.assert_array_equal(xi[1:], one[1:])
    ref = O.xi_tables(k, P, bands, layout)[0]
    assert np.max(np.abs(one[0] - ref)) <= 1e-12 * np.max(np.abs(ref))  # the tables' parity bound

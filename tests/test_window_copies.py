"""The histogram copies and the packed loop of the window kernels: narrow, wide and several-pass
windows, node counts whose canonical pairs are odd in number, a table that ends inside windows."""
import numpy as np
import pytest

from opsec_gpu import api, synth

pytestmark = pytest.mark.gpu

# (linear points, log points, end of the linear section, end of the table)
LAYOUTS = [(256, 4096, 10.0, 20000.0), (64, 300, 10.0, 20000.0), (64, 900, 10.0, 20000.0), (16, 2000, 10.0, 1900.0)]


def _signal(sv, cells, layout, gauss, extra):
    with api.Engine(api.make_config(sv, bands=synth.band_edges(3, 0.0, 0.3), layout=layout, gauss=gauss,
                                    extra=extra)) as e:
        e.set_pk(*synth.pk_table())
        return [e.signal_block(cells, table=t) for t in (0, 2)]


@pytest.mark.parametrize("gauss", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_packed_loop_has_the_general_loops_bits(layout, gauss):
    sv, cells = synth.shell_survey(5, 6, 20)
    a = _signal(sv, cells, layout, gauss, [])
    b = _signal(sv, cells, layout, gauss, ["cubature.log_keys = 0"])
    for x, y in zip(a, b):
        assert np.all(np.isfinite(x)) and np.array_equal(x, y)


@pytest.mark.parametrize("bins", [16, 44, 48, 52, 100, 384])
@pytest.mark.parametrize("name", ["shell", "box"])
def test_number_of_copies_leaves_the_sums(name, bins):
    """The copies follow the row length; the bins' sums are integers, so the matrix depends on it only where
    the number of passes does: dot products in FP32 chunks (2^-24 of a key's positive sum, a few times over) in
    one, near FP64 in more."""
    sv, cells = synth.shell_survey(5, 6, 20) if name == "shell" else synth.box_survey(6)
    a = _signal(sv, cells, LAYOUTS[1], 4, [])
    b = _signal(sv, cells, LAYOUTS[1], 4, [f"cubature.window_bins = {bins}"])
    for x, y in zip(a, b):
        assert np.max(np.abs(x - y)) <= 1e-6 * np.max(np.abs(x))

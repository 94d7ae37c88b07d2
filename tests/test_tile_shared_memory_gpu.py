"""Handles with large and small tiles side by side: the shared memory that a
tile kernel may take is an attribute of the kernel, shared by every handle of
the process, and a handle made later must not take it from an earlier one."""
import numpy as np
import pytest

import hydrob200 as hb
from hydrob200 import deck as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,large", [("fp32", 1024), ("split", 1024), ("fp64", 512), ("fp64", 1024)])
@pytest.mark.parametrize("small", [64, 0])
def test_large_tiles_step_after_a_small_tile_handle(precision, large, small, tmp_path):
    D.write_deck(D.channel_deck("c", 3000, 3000.0, 900.0, 3, steps=20, dt=0.5), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    first = hb.Solver(deck, precision=precision, layout="tile", tile_cells=large)
    second = hb.Solver(deck, precision=precision, layout="tile", tile_cells=small)
    first.step(3)
    first.capture_graph(4)
    first.graph_launch()
    second.step(7)
    first.sync()
    second.sync()
    a, b = first.get_state(), second.get_state()
    for k in "HUVZW":     # the tile size changes no arithmetic
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    first.close()
    second.close()

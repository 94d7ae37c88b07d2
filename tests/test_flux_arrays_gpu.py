"""The fluxes as they leave and enter a handle: hb_get_flux with some arrays left
out, and a checkpoint's four flux arrays, which a batch moves through a staging
buffer in several pieces, against each other and through a save and a load."""
import ctypes as C

import numpy as np
import pytest

import hydrob200 as hb
from hydrob200 import _lib
from perf.cases import Mesh

pytestmark = pytest.mark.gpu

FLUX = ("FLUX0", "FLUX1", "FLUX2", "FLUX3")


def _checkpoint_fluxes(s, blob, real):
    """The four arrays [4 cells] of a checkpoint, device order: after the header (56 bytes), state and W."""
    n = s.cells
    at = 56 + 5 * n * np.dtype(real).itemsize
    return np.frombuffer(blob, real, 16 * n, at).reshape(4, 4 * n).astype(np.float64)


@pytest.mark.parametrize("precision,real", [("fp64", np.float64), ("split", np.float32)])
@pytest.mark.parametrize("cells", [(900,), (700, 700, 700, 699, 1), (3, 2000)])
def test_fluxes_in_and_out(precision, real, cells):
    meshes = [Mesh("channel", max(n, 8), 3 + i) for i, n in enumerate(cells)]
    make = lambda **kw: hb.Batch(meshes, precision=precision, **kw) if len(meshes) > 1 else hb.Solver(meshes[0], precision=precision, **kw)
    a, b = make(), make(init_state=False)
    a.step(3)
    blob = a.checkpoint()
    b.restore(blob)
    assert b.checkpoint() == blob
    saved = _checkpoint_fluxes(a, blob, real)
    at = 0
    for i, m in enumerate(meshes):
        kw = {"scenario": i} if len(meshes) > 1 else {}
        perm = a.permutation(**kw).astype(np.int64)
        f = a.flux(**kw)
        where = (4 * perm[:, None] + np.arange(4)).reshape(-1)
        for k, name in enumerate(FLUX):
            assert np.any(f[name] != 0.0)
            np.testing.assert_array_equal(f[name][where], saved[k, at:at + 4 * m.cells], err_msg=name)
            only = np.full(4 * m.cells, np.nan)
            ptr = [None] * 4
            ptr[k] = only.ctypes.data_as(_lib._dp)
            _lib.check(_lib.lib().hb_get_flux_at(a._h, i, *ptr))
            np.testing.assert_array_equal(only, f[name])
        at += 4 * m.cells
    a.step(2)
    b.step(2)
    for i in range(len(meshes)):
        kw = {"scenario": i} if len(meshes) > 1 else {}
        x, y = dict(a.get_state(**kw), **a.flux(**kw)), dict(b.get_state(**kw), **b.flux(**kw))
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
    a.close()
    b.close()

"""The drop-in pair on callers' arrays that are not aligned to a cell's four
slots (scalar loads in the update) against the aligned ones (vector loads), bit
for bit, both element types and variants, on a mixed mesh whose slots take the
queue (boundary codes, zero-length slots, wet-dry edges) and the main pass."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shifted(mesh, names, by):
    """Moves the named arrays `by` elements into larger buffers and points the view at them."""
    import torch
    real = C.c_float if mesh.fp32 else C.c_double
    for k in names:
        old = mesh.T[k]
        buf = torch.zeros(old.numel() + 8, dtype=old.dtype, device=old.device)
        new = buf[by:by + old.numel()]
        new.copy_(old)
        mesh.T[k] = new
        part = mesh.view.sides if hasattr(mesh.view.sides, k.upper()) else mesh.view.cells
        setattr(part, k.upper(), C.cast(C.c_void_p(new.data_ptr()), C.POINTER(real)))


@pytest.mark.parametrize("variant", ["H", "F"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mx,my", [(6, 7), (13, 21)])
def test_unaligned_arrays_give_the_same_bits(variant, precision, mx, my, tmp_path):
    import hydrob200 as hb
    from hydrob200 import deck as D
    D.write_deck(D.stress_deck("s", mx, my, 17, steps=12, mdt=13, with_breach=True), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    a = hb.RefLayoutMesh(deck, variant=variant, precision=precision)
    b = hb.RefLayoutMesh(deck, variant=variant, precision=precision)
    _shifted(b, ["FLUX0", "FLUX2", "side", "slsin"], 1)
    a.run(12)
    b.run(12)
    da, db = a.dump(), b.dump()
    for k in da:
        assert np.array_equal(da[k], db[k], equal_nan=True), k

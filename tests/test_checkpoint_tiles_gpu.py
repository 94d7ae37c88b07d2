"""A checkpoint of a handle with balanced tiles (tile_cells = 0, fp32 or split)
loads into one whose tiles were balanced for another number of CTAs per SM, as the
default shape has changed from 3 to 4 per SM: the continued run is the
uninterrupted one bit for bit, fluxes and breached codes included.  A checkpoint of
another mesh of as many cells stays refused."""
import numpy as np
import pytest

import hydrob200 as hb
from hydrob200 import deck as D

pytestmark = pytest.mark.gpu


def _shape(per_sm):
    return next(k for k, s in hb.launch_shapes().items()
                if s["layout"] == "tile" and s["threads"] == 256 and s["min_blocks"] == per_sm)


def _contents(s, n):
    out = []
    for i in range(n):
        kw = {"scenario": i} if n > 1 else {}
        out.append(dict(s.get_state(**kw), **s.flux(**kw), KLAS=s.klas(**kw)))
    return out


@pytest.fixture(scope="module")
def decks(tmp_path_factory):
    out = []
    for name, mx, my, seed in (("wide", 200, 150, 23), ("small", 70, 50, 29)):
        root = str(tmp_path_factory.mktemp(name))
        D.write_deck(D.stress_deck(name, mx, my, seed, steps=10, with_breach=True), root)
        out.append(hb.Deck(root))
    return out


@pytest.mark.parametrize("precision", ["fp32", "split"])
@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("source,target", [(3, 4), (4, 3)])
def test_other_balance(decks, precision, n, source, target):
    def handle(per_sm, init):
        opts = dict(precision=precision, layout="tile", tile_config=_shape(per_sm), init_state=init)
        return hb.Solver(decks[0], **opts) if n == 1 else hb.Batch(decks, **opts)
    a = handle(source, True)
    a.step(1)                                    # the breaching slots are open after it
    blob = a.checkpoint()
    a.step(4)
    a.sync()
    b = handle(target, False)
    perm = [s.permutation(**({"scenario": 0} if n > 1 else {})) for s in (a, b)]
    assert not np.array_equal(*perm)             # the two partitions differ
    b.restore(blob)
    b.step(4)
    b.sync()
    for i, (x, y) in enumerate(zip(_contents(a, n), _contents(b, n))):
        for k in x:
            assert np.array_equal(x[k], y[k], equal_nan=True), (i, k)
    assert np.any(b.klas(**({"scenario": 0} if n > 1 else {})) != decks[0].array("klas"))
    # and back: the target's own checkpoint into the source's partition
    a.restore(b.checkpoint())
    for x, y in zip(_contents(a, n), _contents(b, n)):
        for k in x:
            assert np.array_equal(x[k], y[k], equal_nan=True), k


def test_another_mesh_stays_refused(decks, tmp_path):
    root = str(tmp_path)
    D.write_deck(D.stress_deck("other", 150, 200, 23, steps=10, with_breach=True), root)
    other = hb.Deck(root)
    opts = dict(precision="split", layout="tile")
    a, b = hb.Solver(other, **opts), hb.Solver(decks[0], **opts)
    with pytest.raises(hb.HydroError):
        b.restore(a.checkpoint())

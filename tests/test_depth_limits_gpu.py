"""HM1 and HM2 of other signs and order than a deck's usual 0 < HM1 < HM2: one
CalculateFlux in every form against the CPU oracle's whole branch chain.  The
forms that single out a common case of an edge must leave a side to the chain
wherever the chain takes another branch.

Bound: as in test_common_case_gpu.py, 16 units in the last place (pow differs by
up to 2, taken up to three times in one flux); a wrong branch is off by far more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _states(zbc, hm1, hm2, seed):
    rng = np.random.default_rng(seed)
    n = zbc.size
    up, down = lambda x: np.nextafter(x, np.inf), lambda x: np.nextafter(x, -np.inf)
    h = rng.choice([hm1, up(hm1), down(hm1), hm2, up(hm2), 0.0, 5e-324, 0.5 * (hm1 + hm2), 0.02, 1.0, 2.0, 2.0], n)
    z = zbc + h
    off = rng.integers(0, 8, n)
    z = np.where(off == 0, zbc, np.where(off == 1, zbc - 0.004, np.where(off == 2, zbc + 0.5 * h, z)))
    z = np.where(off == 3, rng.choice(zbc, n), z)          # exactly some cell's bed
    u = rng.choice([0.0, -0.0, 0.4, -0.4, 2.5, -2.5], n)
    v = rng.choice([0.0, -0.0, 0.3, -0.3, 1.0], n)
    return h, u, v, z


def _ulps(a, b):
    with np.errstate(all="ignore"):
        d = np.abs(a - b) / np.spacing(np.maximum(np.abs(a), np.abs(b)))
    same = (a == b) | (np.isnan(a) & np.isnan(b))
    return np.where(same, 0.0, np.where(np.isfinite(d), d, np.inf))


@pytest.mark.parametrize("hm1,hm2", [(0.0, 0.0), (0.0, 0.01), (-0.01, -0.005), (-0.005, 0.0), (-0.005, -0.01), (0.01, 0.001)])
@pytest.mark.parametrize("seed", [1, 2])
def test_fluxes_at_other_depth_limits(hm1, hm2, seed, tmp_path):
    import torch
    import hydrob200 as hb
    from hydrob200 import deck as D
    from oracle.oracle import OracleDeck
    d = D.stress_deck("s", 20, 33, 60 + seed, steps=5, mdt=13, with_unknown=False, hm1=hm1, hm2=hm2)
    d.zbc[:] = np.round(4.0 * d.zbc) / 4.0                  # beds often equal, so that levels meet them
    D.write_deck(d, str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    assert (deck.mesh.hm1, deck.mesh.hm2) == (hm1, hm2)
    h, u, v, z = _states(deck.array("zbc").copy(), hm1, hm2, seed)
    w = np.sqrt(u * u + v * v)
    o = OracleDeck(str(tmp_path))
    for k, a in zip("huvzw", (h, u, v, z, w)):
        o.arr(k)[:] = a
    o.flux(1, 0)
    ref = {k: o.dump()[k] for k in ("FLUX0", "FLUX1", "FLUX2", "FLUX3")}
    m = hb.RefLayoutMesh(deck)
    for k, a in zip("HUVZW", (h, u, v, z, w)):
        m.T[k].copy_(torch.from_numpy(a))
    m.calculate_flux(1, 0)
    got = {"dropin": {k: m.dump()[k] for k in ref}}
    edge2 = [k for k, s in hb.launch_shapes().items() if s["layout"] == "edge"][1]
    for name, opts in (("two kernels", dict(tile_config=edge2)), ("one launch", {}), ("persistent", dict(persistent=True)),
                       ("tiles", dict(layout="tile", tile_cells=64))):
        s = hb.Solver(deck, **opts)
        s.set_state(h, u, v, z, w)
        s.step(1)
        got[name] = s.flux()
        s.close()
    for name, f in got.items():
        for k in ref:
            bad = _ulps(f[k], ref[k])
            assert bad.max() <= 16, (name, k, int(np.argmax(bad)), int((bad > 16).sum()))

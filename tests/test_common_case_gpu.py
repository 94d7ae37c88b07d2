"""The fluxes' common case (slot_common, pair_record, closed_common) at its
edges, against the CPU oracle's whole branch chain: depths at and next to HM1
and HM2, levels at, above and below both beds, still, critical and supercritical
velocities, signed zeros, subnormal, huge and non-finite values, on a mixed mesh
with every boundary code.  One CalculateFlux, by the drop-in call, the two-kernel
step, the one-launch step and the tile step.

Bound: all operations but pow are the oracle's own, rounded the same; pow
differs by up to 2 units in the last place, taken up to three times in one flux
(KLAS 6), so 16 units are allowed; a wrong branch is off by far more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _states(zbc, hm1, hm2, seed, wild):
    rng = np.random.default_rng(seed)
    n = zbc.size
    up = lambda x: np.nextafter(x, np.inf)
    h = rng.choice([hm1, up(hm1), 0.5 * (hm1 + hm2), hm2, up(hm2), 0.02, 0.3, 1.0, 2.0, 2.0, 2.0, 3.7], n)
    z = zbc + h
    off = rng.integers(0, 10, n)
    z = np.where(off == 0, zbc, np.where(off == 1, zbc - 0.1, np.where(off == 2, zbc + 0.5 * h, z)))
    z = np.where(off == 3, rng.choice(zbc, n), z)          # exactly some cell's bed
    c = np.sqrt(9.81 * h)
    pick = lambda: rng.choice([0.0, -0.0, 0.4, -0.4, 1.0, -1.0, 2.5, -2.5], n) * np.where(rng.random(n) < 0.3, c, 1.0)
    u, v = pick(), pick()
    calm = rng.random(n) < 0.5                              # enough neighbours that are both in the common case
    h, z = np.where(calm, 2.0, h), np.where(calm, zbc + 2.0, z)
    if wild:
        k = rng.choice(n, n // 12, replace=False)
        h[k[0::4]] = rng.choice([5e-324, 1e-290, 1e150, 1e300, np.inf], k[0::4].size)
        u[k[1::4]] = rng.choice([5e-324, 1e160, -1e200, np.inf, np.nan], k[1::4].size)
        z[k[2::4]] = rng.choice([np.inf, -np.inf, np.nan, 1e300], k[2::4].size)
        v[k[3::4]] = rng.choice([-5e-324, -1e160, -np.inf, np.nan], k[3::4].size)
    return h, u, v, z


def _ulps(a, b):
    """Distance in units of the last place; 0 for equal values and for NaN against NaN."""
    with np.errstate(all="ignore"):
        d = np.abs(a - b) / np.spacing(np.maximum(np.abs(a), np.abs(b)))
    same = (a == b) | (np.isnan(a) & np.isnan(b))
    return np.where(same, 0.0, np.where(np.isfinite(d), d, np.inf))


@pytest.mark.parametrize("wild", [False, True])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_fluxes_at_the_edges_of_the_common_case(seed, wild, tmp_path):
    import torch
    import hydrob200 as hb
    from hydrob200 import deck as D
    from oracle.oracle import OracleDeck
    D.write_deck(D.stress_deck("s", 20, 33, 40 + seed, steps=5, mdt=13, with_unknown=False), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    h, u, v, z = _states(deck.array("zbc").copy(), deck.mesh.hm1, deck.mesh.hm2, seed, wild)
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
    shapes = hb.launch_shapes()
    edge2 = [k for k, s in shapes.items() if s["layout"] == "edge"][1]
    for name, opts in (("two kernels", dict(tile_config=edge2)), ("one launch", {}),
                       ("tiles", dict(layout="tile", tile_cells=64))):
        s = hb.Solver(deck, **opts)
        s.set_state(h, u, v, z, w)
        s.step(1)
        got[name] = s.flux()
        s.close()
    for name, f in got.items():
        for k in ref:
            assert _ulps(f[k], ref[k]).max() <= 16, (name, k, int(np.argmax(_ulps(f[k], ref[k]))))
            assert np.array_equal(f[k].view(np.uint64)[~np.isnan(f[k])],
                                  got["dropin"][k].view(np.uint64)[~np.isnan(f[k])]), (name, k)

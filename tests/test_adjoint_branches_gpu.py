"""The reverse step on a wetting and drying state: a dam break over a rough
bed, whose slots take the dry, shallow, one-sided and supercritical branches
beside the subcritical one, on meshes around a CTA's 32 cells.  Directional
derivatives for n and ZBC against the complex-step reference.  Bound: the two
rollouts differ by the power function's last bits, at most 1e-11 of the state
after these steps (the rollout test's bound); a front's derivatives amplify
that by up to about 1e4.
"""
import numpy as np
import pytest

import hydrob200 as hb
from hydrob200 import deck as D
from hydrob200.adjoint import Adjoint
from oracle import complex_step as CS

pytestmark = pytest.mark.gpu

NSTEPS, OBS_EVERY = 30, 5


@pytest.mark.parametrize("cells,k", [(96, 7), (100, 30), (2500, 10)])
def test_dam_break_gradient_against_complex_step(cells, k, tmp_path):
    side = 30.0 * np.sqrt(cells / 2.0)
    D.write_deck(D.dam_break_deck(cells, side, seed=5 + cells, relief=4.0, level=4.0, dam_x=0.5 * side, steps=NSTEPS),
                 str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    rng = np.random.default_rng(cells)
    gauges = np.sort(rng.choice(deck.cells, min(24, deck.cells // 4), replace=False))
    n0 = np.sqrt(deck.array("fnc") / 9.81).copy()
    zbc = deck.array("zbc").copy()
    a = Adjoint(deck, gauges, OBS_EVERY, NSTEPS, checkpoint_every=k)
    _, obs = a.forward()
    obs = obs + 0.1 * rng.standard_normal(obs.shape)
    a.set_observations(obs)
    L, _ = a.forward()
    gn, gz = a.backward()
    d = CS.ComplexDeck(deck)
    st = deck.state()
    vn, vz = rng.standard_normal(deck.cells), rng.standard_normal(deck.cells)
    for g, dn, dz in ((gn, vn, None), (gz, None, vz)):
        Lc, cs = CS.directional_derivative(d, n0, zbc, st["Z"], st["U"], st["V"], gauges, obs, OBS_EVERY, NSTEPS, dn, dz)
        adj = float(g @ (dn if dn is not None else dz))
        assert abs(Lc - L) <= 1e-9 * abs(L)
        assert abs(adj - cs) <= 1e-7 * abs(cs), (adj, cs)
    a.close()

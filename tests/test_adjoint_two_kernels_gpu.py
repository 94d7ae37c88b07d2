"""The gradient by the two-kernel step (meshes beyond the one-launch step's, or
another edge shape): the recomputed steps' update coefficients, the fused
checkpoints and gauge depths.  Loss, depths and gradient are those of the
one-launch step bit for bit, at checkpoint intervals that divide the steps and
that do not; and just above the one-launch step's size the gradient does not
depend on the interval and equals the complex-step reference's directional
derivative (bound as in test_adjoint_gpu.py, 1e-8).
"""
import numpy as np
import pytest

import hydrob200 as hb
from hydrob200 import deck as D
from hydrob200.adjoint import Adjoint
from oracle import complex_step as CS
from perf.cases import Mesh

pytestmark = pytest.mark.gpu

NSTEPS, OBS_EVERY = 40, 10


def _gradient(deck, gauges, k, nsteps, obs_every, tile_config=0):
    a = Adjoint(deck, gauges, obs_every, nsteps, checkpoint_every=k, tile_config=tile_config)
    rng = np.random.default_rng(3)
    _, obs = a.forward()
    obs = obs + 0.1 * rng.standard_normal(obs.shape)
    a.set_observations(obs)
    L, depths = a.forward()
    gn, gz = a.backward()
    gn2, gz2 = a.backward()                      # the last segment recomputed too
    assert np.array_equal(gn, gn2) and np.array_equal(gz, gz2)
    state = a.solver.get_state()
    a.close()
    return obs, dict(state, L=L, depths=depths, gn=gn, gz=gz)


@pytest.mark.parametrize("k", [10, 7, 40])
@pytest.mark.parametrize("name", ["f1", "dam"])
def test_equals_the_one_launch_step(name, k, tmp_path):
    D.write_deck(D.config_f1(steps=60) if name == "f1" else
                 D.dam_break_deck(2500, 1000.0, seed=8, relief=4.0, level=4.0, dam_x=500.0, steps=60), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    gauges = np.sort(np.random.default_rng(5).choice(deck.cells, 12, replace=False))
    edges = [c for c, s in hb.launch_shapes().items() if s["layout"] == "edge"]
    _, want = _gradient(deck, gauges, k, NSTEPS, OBS_EVERY)
    for shape in edges[:2]:
        _, got = _gradient(deck, gauges, k, NSTEPS, OBS_EVERY, tile_config=shape)
        for q in want:
            np.testing.assert_array_equal(got[q], want[q], err_msg=f"{q}, shape {shape}")


def test_above_the_one_launch_size():
    mesh = Mesh("channel", 34002, 4)
    gauges = np.sort(np.random.default_rng(6).choice(mesh.cells, 30, replace=False))
    obs, want = _gradient(mesh, gauges, 4, 12, 4)
    for k in (5, 12):
        _, got = _gradient(mesh, gauges, k, 12, 4)
        for q in want:
            np.testing.assert_array_equal(got[q], want[q], err_msg=f"{q}, k = {k}")
    d = CS.ComplexDeck(mesh)
    st = mesh.state()
    n0 = np.sqrt(mesh.array("fnc") / 9.81)
    vz = np.random.default_rng(7).standard_normal(mesh.cells)
    Lc, cs = CS.directional_derivative(d, n0, mesh.array("zbc").copy(), st["Z"], st["U"], st["V"], gauges, obs, 4, 12, None, vz)
    assert abs(Lc - want["L"]) <= 1e-9 * abs(want["L"])
    assert abs(float(want["gz"] @ vz) - cs) <= 1e-8 * abs(cs)

"""The persistent kernel where a CTA's flux chunks fill its queue of sides more
than once in a step (more than 8 chunks of 128 records to each resident CTA), so
that the queue is run within the flux phase: bit for bit the two-kernel step, with
most edges queued and with few."""
import numpy as np
import pytest

from perf.cases import HM1, Mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    return Mesh("mixed", 850_001, 3)             # about 10,000 chunks; 592 CTAs at 4 per SM, 888 at 6


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("flow", ["channel", "thin", "patches"])
def test_equals_two_kernels(mesh, precision, flow):
    import hydrob200 as hb
    rng = np.random.default_rng(9)
    n = mesh.cells
    st = mesh.state()
    h, u, v, z = st["H"], st["U"], st["V"], st["Z"]
    if flow == "thin":
        h, u, v = 0.002 + 0.007 * rng.random(n), np.full(n, 0.0005), np.full(n, 0.0002)
        z = mesh.array("zbc") + h
    elif flow == "patches":
        dry = rng.random(n) < 0.5
        h, u, v = np.where(dry, HM1, 0.5), np.where(dry, 0.0, 0.3), np.where(dry, 0.0, 0.1)
        z = mesh.array("zbc") + h
    edge2 = [k for k, s in hb.launch_shapes().items() if s["layout"] == "edge"][1]
    out = []
    for opts in (dict(tile_config=edge2), dict(persistent=True)):
        s = hb.Solver(mesh, precision=precision, **opts)
        s.set_state(h, u, v, z, np.hypot(u, v))
        s.step(3)
        s.sync()
        out.append(dict(s.get_state(), **s.flux()))
        s.close()
    for k in out[0]:
        assert np.array_equal(out[1][k], out[0][k], equal_nan=True), k

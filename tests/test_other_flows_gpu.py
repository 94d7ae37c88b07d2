"""Flows in which most edges lie outside still, subcritical water: supercritical
along and against the edges' direction, a thin sheet (all cells between HM1 and
HM2), wet and dry cells in patches, and depths that jump from cell to cell.  The
sides that the step kernels queue, and those they finish in the main pass, give in
every form what the drop-in pair gives, bit for bit, over some steps."""
import numpy as np
import pytest

from perf.cases import HM1, Mesh

pytestmark = pytest.mark.gpu

STEPS = 6


def _flow(mesh, kind):
    rng = np.random.default_rng(5)
    n = mesh.cells
    h, u, v = 1.0 + 0.05 * rng.random(n), 0.1 * rng.random(n), 0.1 * rng.random(n)
    if kind == "supercritical":
        u += np.where(rng.random(n) < 0.5, 6.0, 5.0)
    elif kind == "against":
        u -= 6.0
        v += 2.0
    elif kind == "thin":
        h, u, v = 0.002 + 0.007 * rng.random(n), 0.0005 + 0 * u, 0.0002 + 0 * v
    elif kind == "patches":
        dry = rng.random(n) < 0.5
        h, u, v = np.where(dry, HM1, 0.5), np.where(dry, 0.0, 0.3), np.where(dry, 0.0, 0.1)
    elif kind == "jumps":
        h = rng.choice([0.5, 0.006, 1.5, 0.02], n)
        u, v = 1.0 + u, v - 0.5
    return h, u, v, mesh.array("zbc") + h


@pytest.mark.parametrize("kind", ["supercritical", "against", "thin", "patches", "jumps"])
@pytest.mark.parametrize("mesh,cells,variant", [("channel", 1201, "H"), ("mixed", 2003, "F")])
def test_every_form_gives_the_drop_in_bits(kind, mesh, cells, variant):
    import hydrob200 as hb
    import torch
    m = Mesh(mesh, cells, 7)
    h, u, v, z = _flow(m, kind)
    w = np.hypot(u, v)
    ref = hb.RefLayoutMesh(m, variant=variant)
    for k, a in zip("HUVZW", (h, u, v, z, w)):
        ref.T[k].copy_(torch.from_numpy(a))
    ref.run(STEPS)
    want = ref.dump()
    edge2 = [k for k, s in hb.launch_shapes().items() if s["layout"] == "edge"][1]
    for name, opts in (("one launch", {}), ("two kernels", dict(tile_config=edge2)), ("persistent", dict(persistent=True)),
                       ("tiles", dict(layout="tile", tile_cells=64)), ("batch", {})):
        s = hb.Batch([m, m], variant=variant, **opts) if name == "batch" else hb.Solver(m, variant=variant, **opts)
        for i in range(2 if name == "batch" else 1):
            s.set_state(h, u, v, z, w, **({"scenario": i} if name == "batch" else {}))
        s.step(STEPS)
        s.sync()
        for i in range(2 if name == "batch" else 1):
            kw = {"scenario": i} if name == "batch" else {}
            got = dict(s.get_state(**kw), **s.flux(**kw))
            for k in got:
                assert np.array_equal(got[k], want[k]), (name, i, k)
        s.close()

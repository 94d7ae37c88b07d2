"""Slots whose code leaves fluxes unwritten (KLAS 13 here: FLUX2 only) keep the
fluxes of the step before (functors.cu:525-565), also those that a supercritical
step, which writes all four, left there in the middle of a sequence of steps.  So a
run does not depend on how its steps are cut into sequences: against the drop-in
pair, which stores every slot's fluxes at every step, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 24


def _bits(a):
    return np.where(np.isnan(a), np.nan, a).view(np.uint64)


@pytest.mark.parametrize("variant", ["H", "F"])
@pytest.mark.parametrize("mx,my,seed", [(8, 9, 3), (12, 17, 4), (20, 33, 9)])
def test_run_does_not_depend_on_the_sequences(variant, mx, my, seed, tmp_path):
    import hydrob200 as hb
    from hydrob200 import deck as D
    D.write_deck(D.stress_deck("s", mx, my, seed, steps=STEPS, mdt=13, with_breach=True), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    # (the drop-in pair's KLAS changes beside the neighbours' reads; a breach here opens at the first step)
    ref = hb.RefLayoutMesh(deck, variant=variant)
    ref.run(STEPS)
    want = ref.dump()
    edge2 = [k for k, s in hb.launch_shapes().items() if s["layout"] == "edge"][1]
    for name, opts in (("one launch", {}), ("two kernels", dict(tile_config=edge2)), ("persistent", dict(persistent=True)),
                       ("tiles", dict(layout="tile", tile_cells=64))):
        for cuts in ((STEPS,), (1, 2, STEPS - 3), (1,) * STEPS):
            s = hb.Solver(deck, variant=variant, **opts)
            for n in cuts:
                s.step(n)
            got = dict(s.get_state(), **s.flux())
            s.close()
            for k in got:
                assert np.array_equal(_bits(got[k]), _bits(want[k])), (name, cuts, k)


@pytest.mark.parametrize("precision,layout", [("fp32", "edge"), ("split", "edge"), ("split", "tile"), ("fp32", "tile")])
def test_cuts_agree_in_the_other_precisions(precision, layout, tmp_path):
    import hydrob200 as hb
    from hydrob200 import deck as D
    D.write_deck(D.stress_deck("s", 12, 17, 4, steps=STEPS, mdt=13), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    runs = []
    for cuts in ((STEPS,), (1, 2, STEPS - 3), (1,) * STEPS):
        s = hb.Solver(deck, precision=precision, layout=layout, tile_cells=64 if layout == "tile" else 0)
        for n in cuts:
            s.step(n)
        runs.append(dict(s.get_state(), **s.flux()))
        s.close()
    for k in runs[0]:
        for r in runs[1:]:
            assert np.array_equal(_bits(r[k]), _bits(runs[0][k])), k

"""The one-launch step of small fp64 meshes against the two-kernel step, bit
for bit: meshes around a CTA's 96 slots and 32 cells (all triangles, mixed,
scattered numbering), every boundary code with a breach that opens on the way,
both variants, single steps and graph replays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 24


def _run(deck, variant, tile_config, graph):
    import hydrob200 as hb
    s = hb.Solver(deck, variant=variant, tile_config=tile_config)
    if graph:
        s.capture_graph(STEPS // 3)
        for _ in range(3):
            s.graph_launch()
    else:
        for n in (1, 2, STEPS - 3):
            s.step(n)
    out = dict(s.get_state(), **s.flux(), KLAS=s.klas())
    s.close()
    return out


def _decks():
    from hydrob200 import deck as D
    yield "tri_94", lambda: D.channel_deck("t", 94, 600.0, 300.0, 5, steps=STEPS, dt=0.5)
    yield "tri_96", lambda: D.channel_deck("t", 96, 600.0, 300.0, 6, steps=STEPS, dt=0.5)
    yield "tri_6675", lambda: D.config_f1(steps=STEPS)
    for mx, my, seed in ((8, 9, 3), (12, 17, 4), (20, 33, 9)):
        yield f"mixed_{mx}x{my}", lambda mx=mx, my=my, seed=seed: D.stress_deck("s", mx, my, seed, steps=STEPS, mdt=13,
                                                                               with_breach=True)
    yield "dam_2500", lambda: D.dam_break_deck(2500, 1500.0, dam_x=750.0, steps=STEPS)


@pytest.mark.parametrize("name", [n for n, _ in _decks()])
@pytest.mark.parametrize("variant", ["H", "F"])
def test_one_launch_step_equals_two_kernels(name, variant, tmp_path):
    import hydrob200 as hb
    from hydrob200 import deck as D
    D.write_deck(dict(_decks())[name](), str(tmp_path))
    deck = hb.Deck(str(tmp_path))
    two_kernels = [k for k, v in hb.launch_shapes().items() if v["layout"] == "edge"][1]
    for graph in (False, True):
        ref = _run(deck, variant, two_kernels, graph)
        got = _run(deck, variant, 0, graph)
        for k in ref:
            assert np.array_equal(got[k].view(np.uint64), ref[k].view(np.uint64)), (k, graph)

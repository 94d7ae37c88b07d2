"""The launch shapes' numbers (tile_config) are published: a number kept from an
earlier hb_autotune or hb_launch_shapes names the same shape in every build.
New shapes are appended."""
import hydrob200 as hb

# number: layout, threads, CTAs per SM of the flux (or tile) kernel, of the cell kernel
SHAPES = {
    1: ("edge", 128, 7, 8), 2: ("edge", 128, 6, 8), 3: ("edge", 128, 8, 8), 4: ("edge", 256, 3, 6),
    5: ("edge", 256, 4, 8), 6: ("edge", 128, 7, 6), 7: ("edge", 256, 2, 6), 8: ("edge", 64, 12, 8),
    9: ("tile", 256, 3, 0), 10: ("tile", 256, 2, 0), 11: ("tile", 128, 6, 0), 12: ("tile", 128, 4, 0),
    13: ("tile", 512, 1, 0), 14: ("tile", 256, 4, 0), 15: ("edge", 128, 6, 6), 16: ("edge", 128, 6, 9),
    17: ("edge", 128, 7, 9), 18: ("tile", 128, 8, 0), 19: ("tile", 256, 5, 0),
}


def test_numbers_name_the_shapes_they_always_named():
    got = hb.launch_shapes()
    for k, want in SHAPES.items():
        s = got[k]
        assert (s["layout"], s["threads"], s["min_blocks"], s["update_min_blocks"]) == want, k

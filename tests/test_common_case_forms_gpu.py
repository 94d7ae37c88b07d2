"""The fluxes' common case (pair_record, slot_common) in every precision, single
and in a batch, against the same edges in the general chain: on a second mesh the
higher-numbered side of every inner edge has a code that is neither 0 nor a
boundary code, which takes the same branches and the same Osher route (mirrored)
but leaves the edge out of the common case.  Depths at and next to HM1 and HM2,
and depths whose celerity lies at the ends of the range in which the constant
quotients need no checks in fp32, 2^-15 and 2^15.

fp64: the same bits.  fp32 and split: the two forms differ by the compiler's
choice of fused products.  With V = |u| + |v| + 2 c and D = V^2 / 9.81 (c of the
largest depth or level difference at the edge) FIL, FIR and the tangents have at
most 6 roundings of at most V, so UA and D's root at most 8 eps V, the piece's
depth at most 0.8 eps V^2 <= 8 eps D, and the four fluxes at most 32 eps times D V
(the first) and D V^2 (the others).  A wrong branch is off by about a tenth of
these.
"""
import numpy as np
import pytest

from perf.cases import Mesh

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24
FLUX = ("FLUX0", "FLUX1", "FLUX2", "FLUX3")


def _mesh(kind, cells, band, general):
    m = Mesh(kind, cells, 11)
    klas, nac = m.arrays["klas"], m.arrays["nac"].astype(int) - 1
    own = np.repeat(np.arange(cells), 4)
    if general:
        klas[(klas == 0.0) & (nac >= 0) & (nac < own)] = 9.0
    if band:                                     # flat bed, thresholds far below
        m.arrays["zbc"][:] = 0.0
        m.mesh.hm1, m.mesh.hm2 = 1e-14, 1e-13
    else:
        m.arrays["zbc"][:] = np.round(4.0 * m.arrays["zbc"]) / 4.0
    return m, nac, own


def _state(m, band, rng):
    n, f = m.cells, np.float32
    near = lambda x: rng.choice([f(x), np.nextafter(f(x), f(9e9)), np.nextafter(f(x), f(0))], n)
    zbc = m.array("zbc")
    if band:
        c = np.float64(2.0) ** band * rng.choice([1.0, 1.0 - 2 * EPS, 1.0 + 2 * EPS, 0.5, 0.9, 1.1, 2.0], n)
        h = f(c * c / 9.81).astype(np.float64)
    else:
        pick = rng.integers(0, 8, n)
        h = np.select([pick == 0, pick == 1, pick == 2, pick == 3],
                      [near(m.mesh.hm1), near(m.mesh.hm2), f(0.02) + 0 * zbc, near(0.3)], f(2.0)).astype(np.float64)
        c = np.sqrt(9.81 * h)
    z = zbc + h
    if not band:
        off = rng.integers(0, 12, n)
        z = np.where(off == 0, zbc, np.where(off == 1, zbc - 0.125, np.where(off == 2, rng.choice(zbc, n), z)))
    speed = lambda: f(c * rng.choice([0.0, 0.1, -0.1, 0.4, -0.4, 1.0, -1.0, 2.5], n)).astype(np.float64)
    return h, speed(), speed(), z


@pytest.mark.parametrize("precision", ["fp64", "fp32", "split"])
@pytest.mark.parametrize("band", [0, -15, 15])
@pytest.mark.parametrize("kind,cells,variant", [("mixed", 1201, "H"), ("channel", 2002, "F")])
def test_forms_against_the_general_chain(precision, band, kind, cells, variant):
    import hydrob200 as hb
    import torch
    m, nac, own = _mesh(kind, cells, band, False)
    g, _, _ = _mesh(kind, cells, band, True)
    h, u, v, z = _state(m, band, np.random.default_rng([cells, band + 20]))
    w = np.hypot(u, v)
    edge2 = [k for k, s in hb.launch_shapes().items() if s["layout"] == "edge"][1]

    def fluxes(mesh, batch=False, **opts):
        s = (hb.Batch([mesh, mesh], precision=precision, variant=variant, **opts) if batch else
             hb.Solver(mesh, precision=precision, variant=variant, **opts))
        for i in range(2 if batch else 1):
            s.set_state(h, u, v, z, w, **({"scenario": i} if batch else {}))
        s.step(1)
        f = s.flux(**({"scenario": 1} if batch else {}))
        s.close()
        return f

    ref = fluxes(g, tile_config=edge2)
    got = {"default": fluxes(m), "two kernels": fluxes(m, tile_config=edge2), "batch": fluxes(m, batch=True),
           "tiles": fluxes(m, layout="tile", tile_cells=64), "batch of tiles": fluxes(m, batch=True, layout="tile", tile_cells=64),
           "persistent": fluxes(m, persistent=True)}
    if precision != "split":
        r = hb.RefLayoutMesh(m, precision=precision, variant=variant)
        for k, a in zip("HUVZW", (h, u, v, z, w)):
            r.T[k].copy_(torch.from_numpy(a))
        r.calculate_flux(1, 0)
        got["dropin"] = {k: np.asarray(r.dump()[k], dtype=np.float64) for k in FLUX}
    nb = np.where(nac >= 0, nac, own)
    zbc = m.array("zbc")
    d = np.max([h[own], h[nb], np.abs(z[nb] - zbc[own]), np.abs(z[own] - zbc[nb])], axis=0)
    V = np.maximum((np.abs(u) + np.abs(v))[own], (np.abs(u) + np.abs(v))[nb]) + 2.0 * np.sqrt(9.81 * d)
    D = V * V / 9.81
    inner = m.array("klas") == 0.0               # (boundary codes are in both meshes the same slots)
    for name, f in got.items():
        for k in FLUX:
            if precision == "fp64":
                assert np.array_equal(f[k], ref[k], equal_nan=True), (name, k)
            else:
                off = np.abs(f[k][inner] - ref[k][inner]) / (32 * EPS * D * V * (1.0 if k == "FLUX0" else V))[inner]
                assert off.max() <= 1.0, (name, k, off.max())

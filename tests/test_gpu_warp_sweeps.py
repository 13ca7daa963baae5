"""The warp-tile H and E sweeps against the plain routines at the sizes where
tiles, vectors and CPML boxes end: widths that leave part of a vector or of a
32-column tile, rows and planes that leave part of a tile, an interior between
the x slabs narrower than a vector, every kind of material ID (PEC, ID 2 with
and without the Drude-Lorentz module, IDs past the staged coefficients).

Tolerance: a step rounds each component about ten times, 6e-8 of it in FP32 and
1.1e-16 in FP64; over 20 steps from fields of order one the two orders of
rounding stay within 1e-5 and 1e-13 of the field's norm."""
import numpy as np
import pytest

from conftest import rel_l2
from cpsfdtd_b200 import decks

pytestmark = pytest.mark.gpu

# nx, ny, nz, CPML cells of the x, y and z axes
SIZES = [(34, 13, 9, 16, 4, 3), (33, 9, 8, 2, 3, 2), (63, 17, 11, 5, 5, 4), (64, 8, 7, 6, 2, 2),
         (67, 14, 10, 7, 3, 3), (97, 31, 25, 9, 9, 9)]


def _deck(nx, ny, nz, pml, dl, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    d = 10e-9
    dk = decks.Deck(nx, ny, nz, d, d, d)
    dk.media = [(1.0 + 0.1 * m, 1.0 + 0.01 * m, 10.0 * m, 5.0 * m) for m in range(24)]
    ids = rng.choice(np.array([0, 0, 0, 1, 2, 3, 4, 15, 16, 23], dtype=np.uint8), size=dk.shape3)
    ids[:, : ny // 2, : nz // 2] = 1  # whole warps of one medium too
    dk.ids = ids.astype(np.uint8)
    dk.pml = decks.pml_params(1)
    dk.pml["npml"] = [pml[0]] * 2 + [pml[1]] * 2 + [pml[2]] * 2
    if dl:
        dk.dl = decks.dl_params_metal()
    fields = []
    for c in range(6):
        f = rng.standard_normal(dk.shape3) * (1.0 if c < 3 else 1.0 / 376.7)
        fields.append(f)
    return dk, fields


@pytest.mark.parametrize("planes", [0, 2, 5, 64])
@pytest.mark.parametrize("dl", [False, True], ids=["id2-idle", "id2-dl"])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_warp_sweeps_equal_plain_routines(prec, dl, planes):
    import cpsfdtd_b200 as cps
    for n, (nx, ny, nz, px, py, pz) in enumerate(SIZES):
        dk, fields = _deck(nx, ny, nz, (px, py, pz), dl, 100 + n)
        out = []
        for path in (cps.PLAIN, cps.FUSED):
            g = cps.Grid.from_deck(dk, prec)
            if path == cps.FUSED and planes:
                g.set_tile(4, planes)
            for c, f in enumerate(fields):
                g.set_field(c, f)
            g.step(20, path)
            g.sync()
            out.append([g.field(c) for c in range(6)])
            g.close()
        for c in range(6):
            err = rel_l2(out[1][c], out[0][c])
            assert err < (1e-13 if prec == 0 else 1e-5), f"{nx}x{ny}x{nz} component {c}: {err:.2e}"

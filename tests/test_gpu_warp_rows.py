"""The warp-tile sweeps on tiles of eight rows, which have their own ring, boxes
and instantiations: the sizes, decks and bounds of test_gpu_warp_sweeps.py
(20 steps, about ten roundings a step and component: 1e-5 of a field's norm in
FP32, 1e-13 in FP64), with and without CPML."""
import pytest

from conftest import rel_l2
from test_gpu_warp_sweeps import SIZES, _deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes", [1, 2, 5, 64])
@pytest.mark.parametrize("dl", [False, True], ids=["id2-idle", "id2-dl"])
@pytest.mark.parametrize("pml", [True, False], ids=["cpml", "open"])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_eight_row_tiles_equal_plain_routines(prec, pml, dl, planes):
    import cpsfdtd_b200 as cps
    for n, (nx, ny, nz, px, py, pz) in enumerate(SIZES):
        dk, fields = _deck(nx, ny, nz, (px, py, pz), dl, 100 + n)
        if not pml:
            dk.pml = None
        out = []
        for path in (cps.PLAIN, cps.FUSED):
            g = cps.Grid.from_deck(dk, prec)
            if path == cps.FUSED:
                g.set_tile(8, planes)
            for c, f in enumerate(fields):
                g.set_field(c, f)
            g.step(20, path)
            g.sync()
            out.append([g.field(c) for c in range(6)])
            g.close()
        for c in range(6):
            err = rel_l2(out[1][c], out[0][c])
            assert err < (1e-13 if prec == 0 else 1e-5), f"{nx}x{ny}x{nz} component {c}: {err:.2e}"

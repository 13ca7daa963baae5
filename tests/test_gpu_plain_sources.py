"""Sources beside the CPML slabs on the plain path.

A step adds its sources between the E bulk update and the E CPML routine
(main.cpp:267-344).  The CPML of an E cell reads H at the cell and one cell
below on each axis, so an H source may reach it from one cell in front of a
far slab; the step then has to keep the two routines apart.  The routines
called one by one are the yardstick: the same operations in the same order,
equal bit for bit."""
import time

import numpy as np
import pytest

from cpsfdtd_b200 import decks
from test_gpu_step_paths import _noise, _same, _state, _tfsf_deck

pytestmark = pytest.mark.gpu


# order of the CPML grading: with 0 the slab's outermost E plane is graded as its
# others (with any other order its psi coefficient is zero)
@pytest.mark.parametrize("m", [0, 3])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_sources_beside_a_slab_equal_the_routines(prec, axis, m):
    import cpsfdtd_b200 as cps
    dk = _tfsf_deck(9)
    dk.pml["m"] = m
    n, np_ = (dk.nx, dk.ny, dk.nz)[axis], dk.pml["npml"][2 * axis]
    wave = 1.0 + 0.25 * np.arange(40.0)
    for at in (np_, np_ + 1, n - np_ - 1, n - np_):
        for comp in range(6):
            p = [18, 12, 16]
            p[axis] = at
            dk.sources = [(comp, *p, wave)]
            a, b = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
            for g in (a, b):
                _noise(g, dk, 5)
            a.step(6, cps.PLAIN)
            n0 = b.get_step()
            for s in range(n0, n0 + 6):
                b.op("h_bulk")
                b.op("tfsf_h", s, 0x3F)
                b.op("h_pml")
                b.op("e_bulk")
                b.op("tfsf_e", s, 0x3F)
                b.op("sources", s)
                b.op("e_pml")
            _same(_state(a), _state(b))
            a.close()
            b.close()


def test_plain_calls_do_not_walk_the_sources():
    """One step at a time costs what steps in one call cost, however many
    sources there are: 50 calls with 200 000 sources, where a walk over them
    takes milliseconds a call and a step's launches under a tenth of one."""
    import cpsfdtd_b200 as cps
    n, d = 72, 5e-9
    dk = decks.Deck(n, n, n, d, d, d)
    dk.pml = decks.pml_params(4)
    g = cps.Grid.from_deck(dk, cps.FP32)
    k, j, i = np.meshgrid(*[np.arange(7, 66)] * 3, indexing="ij")
    at = np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1)[:200000]
    wave = np.ones(1)
    for p in at.tolist():
        g.source_add(decks.COMP["Ez"], *p, wave)

    def ms(calls, steps):
        best = 1e9
        for _ in range(3):
            g.sync()
            t0 = time.perf_counter()
            for _ in range(calls):
                g.step(steps, cps.PLAIN)
            g.sync()
            best = min(best, 1e3 * (time.perf_counter() - t0))
        return best

    ms(1, 2)
    one, many = ms(1, 50), ms(50, 1)
    assert many < one + 25.0, (one, many)

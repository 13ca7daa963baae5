"""Fused steps as replayed chunks after something else has touched the grid:
port samples taken outside the step, media set again, tiles set again, the
wait's test setting, and short calls.  Chunks and single launches do the same
operations on every cell and sample, so results are equal bit for bit."""
import time

import numpy as np
import pytest

from cpsfdtd_b200 import decks
from test_gpu_step_paths import _noise, _same, _state

pytestmark = pytest.mark.gpu


def _pair(dk, prec):
    """the grid in chunks and the same grid in single launches"""
    import cpsfdtd_b200 as cps
    a, b = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
    b.set_chunked(False)
    for g in (a, b):
        _noise(g, dk, 11)
    return a, b


@pytest.mark.parametrize("deck", ["dispersive", "laser"])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_tile_set_on_a_batch_member_between_steps(prec, deck):
    """A member's tile set while it is in a batch whose tables are made: the
    batch's rows hold for its own sweeps (the tensor maps' rows), in chunks
    launched directly (a new length) and replayed (a length that comes again)."""
    import cpsfdtd_b200 as cps
    mk = {"dispersive": lambda n: decks.config2(n=n, steps=1, nfreq=3),
          "laser": lambda n: decks.config4_member(n, n - 3, n - 5, seed=3, steps=1, nfreq=2)}[deck]
    dks = [mk(40), mk(53)]
    got = []
    for tiles in (False, True):
        gs = [cps.Grid.from_deck(dk, prec) for dk in dks]
        for g, dk in zip(gs, dks):
            _noise(g, dk, 12)
        bt = cps.Batch(prec)
        for g in gs:
            bt.add(g)
        for rows, planes in ((8, 8), (4, 8), (8, 16), (4, 2), (8, 1)):
            for n in (7, 12, 12):
                bt.step(n)
                if tiles:
                    gs[0].set_tile(rows, planes)
        bt.sync()
        got.append([_state(g) for g in gs])
        for g in gs:
            bt.remove(g)
        bt.close()
    for x, y in zip(*got):
        _same(x, y)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_tile_set_on_a_chunked_grid(prec):
    """The grid's own chunks follow its tile: rows and planes, the default's own
    among them."""
    import cpsfdtd_b200 as cps
    a, b = _pair(decks.config2(n=45, steps=1, nfreq=3), prec)
    for g in (a, b):
        g.step(192, cps.FUSED)
        for rows, planes in ((4, 8), (8, 8), (8, 1), (4, 64), (16, 4), (4, 8)):
            g.set_tile(rows, planes)
            g.step(64, cps.FUSED)
    _same(_state(a), _state(b))


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_steps_alone_between_batch_steps(prec):
    """A member's own long calls (its own chunks) between the batch's."""
    import cpsfdtd_b200 as cps
    dks = [decks.config2(n=40, steps=1, nfreq=3), decks.config2(n=49, steps=1, nfreq=2)]
    out = []
    for alone in (False, True):
        gs = [cps.Grid.from_deck(dk, prec) for dk in dks]
        for g, dk in zip(gs, dks):
            _noise(g, dk, 13)
        bt = cps.Batch(prec)
        for g in gs:
            bt.add(g)
        for n in (64, 40, 64, 5, 64):
            bt.step(n)
            if alone:
                gs[0].step(70, cps.FUSED)
                gs[0].step(3, cps.FUSED)
        bt.sync()
        if not alone:
            gs[0].step(5 * 73, cps.FUSED)
        out.append([_state(g) for g in gs])
        for g in gs:
            bt.remove(g)
        bt.close()
    for x, y in zip(*out):
        _same(x, y)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_port_samples_between_chunks_are_kept(prec):
    import cpsfdtd_b200 as cps
    dk = decks.config2(n=41, steps=1, nfreq=3)
    a, b = _pair(dk, prec)
    for g in (a, b):
        g.step(64, cps.FUSED)
        n = g.get_step()
        for s in range(n, n + 64):  # a whole ring, the grid's own step number unmoved
            for p in range(len(g.ports)):
                g.op("port_sample", p, s)
        g.step(64, cps.FUSED)
    _same(_state(a), _state(b))


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_media_set_again_reach_the_chunks(prec):
    """ID 2 without the Drude-Lorentz module keeps its E bulk update out, and its
    CPML term takes the medium's curl coefficient: set between two chunks of
    one length, the second of them a replay."""
    import cpsfdtd_b200 as cps
    d = 10e-9
    dk = decks.Deck(40, 37, 33, d, d, d)
    dk.media = [(1.0, 1.0, 0.0, 0.0), (2.25, 1.0, 0.0, 0.0), (2.0, 1.0, 0.0, 0.0)]
    ids = np.zeros(dk.shape3, dtype=np.uint8)
    ids[2:4, 10:14, 12:15] = 2  # in the x slab; such cells only sum psi terms: few steps
    dk.ids = ids
    dk.pml = decks.pml_params(5)
    a, b = _pair(dk, prec)
    for g in (a, b):
        for _ in range(3):
            g.step(32, cps.FUSED)
        g.set_media([(1.0, 1.0, 0.0, 0.0), (2.25, 1.0, 0.0, 0.0), (5.0, 1.0, 0.0, 0.0)])
        g.step(32, cps.FUSED)
    _same(_state(a), _state(b))


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_wait_setting_reaches_the_chunks(prec):
    """A chunk gives up its waits, says so, and the grid steps as a fresh one after
    a reset (no fault is involved: every wait is bounded and every copy lands).
    A grid of 4 Mi cells steps in chunks always; tiles of all its planes are
    few enough to wait at the same time."""
    import cpsfdtd_b200 as cps
    d = 10e-9
    dk = decks.Deck(512, 128, 65, d, d, d)
    dk.sources = [(decks.COMP["Ez"], 250, 64, 30, decks.gaussian_sine(400, dk.dt, 600e-9, 5e-16, 7e-16))]
    g, ref = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
    for q in (g, ref):
        q.set_tile(8, 128)
    g.step(64, cps.FUSED)
    g.sync()
    g.set_wait_skew(256)
    t0 = time.perf_counter()
    g.step(1, cps.FUSED)
    with pytest.raises(cps.CpsError) as ex:
        g.sync()
    assert ex.value.code == cps.CPS_E_TIMEOUT
    assert time.perf_counter() - t0 < 30.0
    g.set_wait_skew(0)
    g.reset(dk.n0)
    for q in (g, ref):
        q.step(64, cps.FUSED)
        q.sync()
    for c in range(6):
        assert np.array_equal(g.field(c), ref.field(c))


def test_short_calls_fold_the_ports_once_a_ring():
    """A loop of single steps on a small grid with a port DFT launches what it does
    on a grid without chunks: the contraction runs once in 64 samples, not once a
    call."""
    import cpsfdtd_b200 as cps
    dk = decks.config2(n=41, steps=1, nfreq=3)
    a, b = _pair(dk, cps.FP32)
    n = []
    for g in (a, b):
        g.step(64, cps.FUSED)
        n0 = g.launches()
        for _ in range(130):
            g.step(1, cps.FUSED)
        n.append(g.launches() - n0)
    assert n[0] <= n[1] + 4, n
    _same(_state(a), _state(b))

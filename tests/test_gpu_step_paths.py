"""One step's work in different launches: the plain path against its routines
called one by one (the CPML boxes of a side as one launch, or as part of the
bulk update's where no injection or source lies in a slab), and small grids'
fused steps as replayed graph chunks, in ragged pieces, against one launch
after another.  The same operations in the same order on each cell, so both
are equal bit for bit."""
import numpy as np
import pytest

from conftest import rel_l2
from cpsfdtd_b200 import decks

pytestmark = pytest.mark.gpu


def _tfsf_deck(inset):
    """TF/SF box `inset` cells inside, CPML of unequal depths, a source."""
    nx, ny, nz, d = 37, 29, 33, 5e-9
    dk = decks.Deck(nx, ny, nz, d, d, d)
    dk.media = [(1.0, 1.0, 0.0, 0.0), (2.25, 1.0, 0.0, 0.0), (1.0, 1.0, 0.0, 0.0)]
    ids = np.zeros(dk.shape3, dtype=np.uint8)
    ids[12:20, 10:16, 11:19] = 1
    dk.ids = ids
    dk.pml = decks.pml_params(1)
    dk.pml["npml"] = [5, 5, 3, 3, 4, 4]
    dk.tfsf = {"lambda": 550e-9, "dlambda": decks.dlambda_for_tau(550e-9, 2e-15), "w0": 100e-9, "z0_deck": 0.0,
               "xs": (nx / 2 + 0.5) * d, "ys": (ny / 2 + 0.5) * d, "zs": 0.0, "k0": nz // 2, "theta": 30.0,
               "phi": 45.0, "E0": 1.0, "psi": 0.0, "n6": [inset] * 6, "Nt": 400, "cwmode": 0}
    return dk


def _sourced(dk, at):
    dk.sources = [(decks.COMP["Ez"], *at, decks.gaussian_sine(400, dk.dt, 600e-9, 5e-16, 7e-16)),
                  (decks.COMP["Ex"], 15, 14, 16, decks.gaussian_sine(30, dk.dt, 500e-9, 4e-16, 5e-16))]
    return dk
    return dk


_DECKS = {
    "clear": lambda: _sourced(_tfsf_deck(9), (18, 12, 16)),
    "box-meets-slab": lambda: _sourced(_tfsf_deck(5), (18, 12, 16)),
    "source-in-slab": lambda: _sourced(_tfsf_deck(9), (3, 12, 16)),
    "source-at-slab-edge": lambda: _sourced(_tfsf_deck(9), (18, 12, 28)),
    "dispersive": lambda: decks.config2(n=41, steps=1, nfreq=3),
    "laser": lambda: decks.config4_member(40, 33, 36, seed=3, steps=1, nfreq=2),
}


def _state(g):
    return [g.field(c) for c in range(6)] + [g.port_last(p) for p in range(len(g.ports))] + [
        g.port_dft(p, raw=True).copy() for p in range(len(g.ports)) if g.ports[p][2] > 0]


def _same(a, b):
    assert np.abs(a[2]).max() > 0
    for q, (x, y) in enumerate(zip(a, b)):
        assert np.array_equal(x, y), (q, rel_l2(x, y))


def _noise(g, dk, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    for c in range(6):
        g.set_field(c, rng.standard_normal(dk.shape3) * (1.0 if c < 3 else 1.0 / 376.7))


@pytest.mark.parametrize("name", list(_DECKS))
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_plain_step_equals_its_routines(name, prec):
    import cpsfdtd_b200 as cps
    dk = _DECKS[name]()
    a, b = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
    for g in (a, b):
        _noise(g, dk, 5)
    a.step(12, cps.PLAIN)
    b.set_record(False)
    n0 = b.get_step()
    for n in range(n0, n0 + 12):
        b.op("h_bulk")
        if dk.tfsf:
            b.op("tfsf_h", n, 0x3F)
        b.op("h_pml")
        b.op("e_bulk")
        if dk.dl:
            b.op("dl")
        if dk.gain:
            for q in ("gain_polarization", "gain_efield", "gain_populations"):
                b.op(q)
        if dk.tfsf:
            b.op("tfsf_e", n, 0x3F)
        if dk.sources:
            b.op("sources", n)
        b.op("e_pml")
        for p in range(len(b.ports)):
            b.op("port_sample", p, n)
    _same(_state(a), _state(b))


@pytest.mark.parametrize("name", list(_DECKS))
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_small_grids_chunks_equal_single_launches(name, prec):
    import cpsfdtd_b200 as cps
    dk = _DECKS[name]()
    a, b = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
    b.set_chunked(False)
    for g in (a, b):
        _noise(g, dk, 6)
        g.step(5, cps.FUSED)    # single launches on both
        g.step(100, cps.FUSED)  # chunks of 64 and 36
        g.step(1, cps.FUSED)
        g.step(2, cps.PLAIN)    # the step number moves outside the chunks
        g.step(67, cps.FUSED)
    _same(_state(a), _state(b))


@pytest.mark.parametrize("planes", [0, 1, 3, 64])
@pytest.mark.parametrize("rows", [4, 8])
def test_fp64_gain_sweep_equals_plain_routines(rows, planes):
    """Gain cells in whole, broken and single-cell runs of a row, in and out of
    the CPML slabs, list groups that start at every offset.  About 40 roundings
    of 1.1e-16 a step over 20 steps stay below 1e-13 of a field's norm; the
    divisions by constants add one each: 1e-12 with room for the recursion."""
    import cpsfdtd_b200 as cps
    for n, (nx, ny, nz, npml) in enumerate([(34, 13, 9, 2), (67, 14, 11, 4), (96, 17, 8, 3)]):
        rng = np.random.Generator(np.random.PCG64(40 + n))
        d = 10e-9
        dk = decks.Deck(nx, ny, nz, d, d, d)
        dk.media = [(1.0 + 0.1 * m, 1.0, 0.0, 0.0) for m in range(24)]
        ids = rng.choice(np.array([0, 1, 4, 5, 5, 5, 17, 23], dtype=np.uint8), size=dk.shape3)
        ids[:, ny // 2:, : nz // 2] = 5
        dk.ids = ids
        dk.pml = decks.pml_params(npml)
        dk.gain = decks.gain_params_laser()
        out = []
        for path in (cps.PLAIN, cps.FUSED):
            g = cps.Grid.from_deck(dk, cps.FP64)
            if path == cps.FUSED:
                g.set_tile(rows, planes or 8)
            _noise(g, dk, 9 + n)
            g.step(20, path)
            out.append([g.field(c) for c in range(6)] + [np.asarray(g.populations())])
            g.close()
        for q, (x, y) in enumerate(zip(*out)):
            assert rel_l2(y, x) < 1e-12, (nx, q, rel_l2(y, x))


@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nfreq", [1, 4, 5, 8, 9, 16, 17, 33])
def test_port_dft_tiles(nfreq, prec, chunked):
    """Ports whose points and frequencies end inside, at and past a tile of the
    contraction, over a whole ring and part of one, against sums of the samples
    in the same precision.  70 terms of one size each: 70 roundings of the sum
    and as many of the phase, 1.1e-16 each, within 1e-12 of the largest."""
    import cpsfdtd_b200 as cps
    n, d, steps = 48, 10e-9, 70
    dk = decks.Deck(n, n, 12, d, d, d)
    dk.media = [(1.0, 1.0, 0.0, 0.0)]
    freqs = np.linspace(0.8, 1.2, nfreq) * 5e14
    for w, h in ((1, 1), (15, 17), (16, 16), (27, 19), (32, 32), (25, 41)):
        dk.ports.append(decks.Port("plain", dict(dir="z", position=6.5 * d, w1=2.5 * d, w2=(2 + w - 0.5) * d,
                                                 h1=3.5 * d, h2=(3 + h - 0.5) * d), dft_freqs=freqs, dft_mask=0x2B))
    a, b = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
    for g in (a, b):
        _noise(g, dk, 3)
        g.set_chunked(chunked)
    n0 = a.get_step()
    a.step(steps, cps.FUSED)
    series = [[] for _ in dk.ports]
    for _ in range(steps):
        b.step(1, cps.FUSED)
        for p in range(len(dk.ports)):
            series[p].append(np.asarray(b.port_last(p)).T)
    comps = [c for c in range(6) if 0x2B >> c & 1]
    for p in range(len(dk.ports)):
        got = np.asarray(a.port_dft(p, raw=True))
        npts = series[p][0].shape[1]
        got = got.reshape(len(comps), nfreq, 2, npts)
        t = (n0 + np.arange(steps)) * dk.dt
        for q, c in enumerate(comps):
            s = np.stack([x[c] for x in series[p]])
            ph = np.outer(2 * np.pi * freqs, t - (0.5 * dk.dt if c >= 3 else 0.0))
            want = np.stack([np.cos(ph) @ s, -np.sin(ph) @ s], axis=1)
            assert np.abs(got[q] - want).max() <= 1e-12 * np.abs(s).sum(axis=0).max(), (p, c)

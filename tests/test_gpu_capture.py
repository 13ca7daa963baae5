"""Steps captured on the caller's stream into the caller's CUDA graph."""
import ctypes as C

import numpy as np
import pytest

from cpsfdtd_b200 import decks
from test_gpu_step_paths import _noise, _same

pytestmark = pytest.mark.gpu

_CASES = {"warm chunks": (64, 40), "first long call": (2, 40), "one step": (64, 1)}


def _deck(n):
    """no TF/SF, sources or ports: their step numbers are arguments of a launch,
    and a replay is to be the same steps again"""
    dk = decks.config2(n=n, steps=1, nfreq=2)
    dk.tfsf, dk.sources, dk.ports = None, [], []
    return dk


@pytest.mark.parametrize("path", [0, 1], ids=["plain", "fused"])
@pytest.mark.parametrize("name", list(_CASES))
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_steps_in_a_callers_graph(prec, name, path):
    import torch

    import cpsfdtd_b200 as cps
    warm, steps = _CASES[name]
    dk = _deck(45)
    a, b = cps.Grid.from_deck(dk, prec), cps.Grid.from_deck(dk, prec)
    b.set_chunked(False)
    for g in (a, b):
        _noise(g, dk, 21)
        g.step(warm, path)
        g.sync()
    s = torch.cuda.Stream()
    assert a.L.cps_grid_set_stream(a.h, C.c_void_p(s.cuda_stream)) == 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            a.step(steps, path)
        finally:
            graph.capture_end()
        for _ in range(3):
            graph.replay()
    s.synchronize()
    b.step(3 * steps, path)
    _same([a.field(c) for c in range(6)], [b.field(c) for c in range(6)])
    # outside a capture the grid goes on as it did
    for g in (a, b):
        g.step(70, path)
    _same([a.field(c) for c in range(6)], [b.field(c) for c in range(6)])

"""Fused steps where device memory is used up: the tables of a grid's chunks do
not fit and the steps are launched one after another, as they were before the
grid had any chunk.  The memory is a pool of limited size, set in a process of
its own, so nothing on the device runs out."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from cuda.bindings import runtime as rt
import cpsfdtd_b200 as cps
from cpsfdtd_b200 import decks


def ok(r):
    assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
    return r[1] if len(r) > 1 else None


d = 10e-9
dk = decks.Deck(40, 37, 33, d, d, d)
dk.pml = decks.pml_params(5)
dk.sources = [(decks.COMP["Ez"], 20, 18, 16, decks.gaussian_sine(400, dk.dt, 600e-9, 5e-16, 7e-16))]
ref = cps.Grid.from_deck(dk, cps.FP32)
ref.set_chunked(False)
ref.step(2 + 70, cps.FUSED)
want = [ref.field(c) for c in range(6)]

props = rt.cudaMemPoolProps()
props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
props.location.id = 0
props.maxSize = 128 << 20
pool = ok(rt.cudaMemPoolCreate(props))
ok(rt.cudaDeviceSetMemPool(0, pool))
g = cps.Grid.from_deck(dk, cps.FP32)
g.step(2, cps.FUSED)
g.field(0)  # the read-out's own buffer
g.sync()
stream = ok(rt.cudaStreamCreate())
n = 64 << 20
while n >= 256:
    r = rt.cudaMallocAsync(n, stream)
    if r[0] != rt.cudaError_t.cudaSuccess:
        rt.cudaGetLastError()
        n //= 2
ok(rt.cudaStreamSynchronize(stream))
assert rt.cudaMallocAsync(1 << 12, stream)[0] == rt.cudaError_t.cudaErrorMemoryAllocation
rt.cudaGetLastError()
g.step(70, cps.FUSED)
g.sync()
for c in range(6):
    assert np.array_equal(g.field(c), want[c]), c
print("same")
"""


def test_steps_go_on_without_room_for_tables():
    r = subprocess.run([sys.executable, "-c", _CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr

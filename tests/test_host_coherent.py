"""Loads of kernels that start before their predecessor ends (pdl.cuh).

The non-coherent load (__ldg) is for words nobody writes while the kernel
lives, and the compiler may move it across the device-side wait.  A kernel of
a step that is launched early lives while its predecessor still writes fields
and psi words, so it reads those with plain loads, which the wait orders;
__ldcg is held to the same rule.  Looked for in the sources, on the CPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpsfdtd_b200", "csrc")
# the early kernels and the bodies they are made of (the register sweeps of
# kernels_fused.cu and the one-pass step start after their predecessor's end)
SOURCES = ["kernels_tma.cu", "tma_bodies.cuh", "warp_tiles.cuh", "kernels_plain.cu", "kernels_ports.cu"]
WRITTEN = re.compile(r"__ld(g|cg|ca|cs|lu|cv)\s*\([^;]*?(\b\w+\.[EH][xyz]\b|\bq[eh]\s*\[)")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def _function(text, name):
    """the body of the function `name`"""
    at = text.index(name + "(")
    at = text.index("{", at)
    depth = 0
    for q in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[q], 0)
        if depth == 0:
            return text[at:q]
    raise AssertionError(name)


def test_early_kernels_read_written_words_with_plain_loads():
    bad = []
    for name in SOURCES:
        code = _code(name)
        bad += [(name, m.group(0)) for m in WRITTEN.finditer(code)]
        assert "__ldcg" not in code, name
    cells = _code("sweep_cells.cuh")
    for fn in ("psi_load_e", "psi_load_h", "gain_fetch64"):
        bad += [(fn, m) for m in re.findall(r"__ld\w+\s*\([^;]*", _function(cells, fn))]
    assert not bad, bad

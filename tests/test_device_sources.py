"""CPU checks of the device sources for what no run shows reliably.

``bar.sync``, ``bar.red`` and the ``tcgen05`` allocation are warp-aligned instructions: a warp whose lanes reach them apart is
undefined behaviour.  Their wrappers are called straight after code that branches by lane, so each has to converge the
warp itself."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gcorr_gb300", "csrc")
ALIGNED = re.compile(r"\b(bar\.sync|bar\.red|barrier\.(cta\.)?(sync|red)\S*\.aligned|tcgen05\.alloc)\b")


def _functions(text):
    """(name, body) of every brace-delimited function of a source."""
    for m in re.finditer(r"(\w+)\s*\([^;{}()]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


def _aligned_wrappers():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as h:
                text = re.sub(r"//[^\n]*", "", h.read())
            out += [(f, name, body) for name, body in _functions(text) if ALIGNED.search(body) and len(body) < 1500]
    return out


def test_every_aligned_instruction_is_in_a_wrapper():
    assert {n for _, n, _ in _aligned_wrappers()} >= {"group_sync", "group_sync_and", "tmem_alloc"}


@pytest.mark.parametrize("file,name,body", _aligned_wrappers(), ids=lambda v: v if isinstance(v, str) and len(v) < 40 else "")
def test_warp_converges_before_an_aligned_instruction(file, name, body):
    assert "__syncwarp();" in body[:ALIGNED.search(body).start()], f"{file}: {name}"


def test_every_shared_device_helper_has_a_caller():
    """The helpers and constants of tcgen05_util.cuh, and the constants of the F-stage sources, are used."""
    text = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as h:
                text[f] = re.sub(r"//[^\n]*", "", h.read())
    names = re.findall(r"__device__ __forceinline__ \w+ (\w+)\(", text["tcgen05_util.cuh"])
    unused = [n for n in names if len(re.findall(r"\b%s\b" % n, "".join(text.values()))) < 2]
    for f, t in text.items():
        unused += [f + ": " + n for n in re.findall(r"\bconstexpr (?:int|float|double|uint32_t) (\w+) =", t)
                   if len(re.findall(r"\b%s\b" % n, "".join(text.values()) if f.endswith(".cuh") else t)) < 2]
    assert not unused

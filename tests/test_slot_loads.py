"""The kernels of a row-slot chain may start while the kernel before them still
writes what they read (programmatic stream serialization), so dvg_slots.cu must
not read through the read-only path: CUDA allows __ldg and const __restrict__
only for memory that nothing writes from the kernel's start to its end.  The
input's ranges, complete before a chain starts, are the one exception
(load_range in k_crs_to_slots)."""
import os
import re

from conftest import ROOT

SOURCE = os.path.join(ROOT, "diverg_b200", "csrc", "dvg_slots.cu")


def code():
    with open(SOURCE) as f:
        text = f.read()
    return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", text), flags=re.S)


def test_chain_kernels_are_launched_close():
    # what the rule below is there for
    assert "cudaLaunchAttributeProgrammaticStreamSerialization" in code()


def test_no_read_only_loads_of_what_a_chain_writes():
    text = code()
    for word in ("__ldg", "__restrict__", "ld.global.nc", "__ldlu"):
        assert word not in text, word
    reads = re.findall(r"load_range\(([^,]+),", text)
    assert reads == ["part.entries"]


def test_every_kernel_waits_before_it_touches_memory():
    # (the wait is the first statement of each kernel, before any load)
    bodies = re.findall(r"__global__ void (?:__launch_bounds__\([^)]*\) )?(\w+)\([^{]*\)\s*\{\s*(\w+)", code())
    assert len(bodies) >= 6
    for name, first in bodies:
        assert first == "follow", name

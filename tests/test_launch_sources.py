"""Kernels that may be started while the one before them still runs (moe_run, moe_common.cuh) read what that one writes
and write what it reads.  `__ldg` promises data that is constant for the kernel's lifetime and `__restrict__` that nothing
else touches the object, so a compiler may move such accesses in front of the wait; these kernels therefore use plain loads
and plain pointers.  A property of the source text, checked as one."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "r-mda_b200", "csrc")


def _strip(text):
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _functions(text):
    """name -> (parameters, body) of every __global__ definition."""
    out = {}
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(1)] = (m.group(2), text[m.end():i])
    return out


SOURCES = {os.path.basename(f): _strip(open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}
KERNELS = {k: (f, *v) for f, t in SOURCES.items() for k, v in _functions(t).items()}
EARLY = sorted({m for t in SOURCES.values() for m in re.findall(r"moe_run\(c,\s*(\w+)", t) + re.findall(r"cudaLaunchKernelEx\(&cfg,\s*(\w+)", t)
                if m != "kernel"})


def test_every_early_kernel_is_found():
    assert len(EARLY) >= 15 and "moe_mm_ws_kernel" in EARLY and set(EARLY) <= set(KERNELS)


@pytest.mark.parametrize("name", EARLY)
def test_early_kernel_waits_and_loads_plainly(name):
    source, params, body = KERNELS[name]
    assert "moe_pdl_begin();" in body
    assert "__restrict__" not in params
    helpers = [] if source == "moe_ep.cu" else [SOURCES[source]]   # that one also holds kernels of serial launches
    for text in [body, SOURCES["moe_common.cuh"], SOURCES["moe_tc.cuh"]] + helpers:
        assert "__ldg(" not in text and "global.nc" not in text

"""Kernels started by launch_pdl run their first instructions while the kernel
before them still writes: each begins with the wait, before any other
statement, and none has a __restrict__ pointer parameter (which would allow
non-coherent loads, or a load moved up across the wait)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blobs_gb300", "csrc")


def sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, f)) as src:
                text = re.sub(r"//[^\n]*|/\*.*?\*/", "", src.read(), flags=re.S)
            yield f, text


def kernels(text):
    """(name, parameters, start of the body) of every kernel defined in text."""
    for m in re.finditer(r"__global__ void(?:\s+__launch_bounds__\([^)]*\))?\s+(\w+)\(([^{;]*)\)\s*\{([^;}]*;)", text):
        yield m.group(1), m.group(2), m.group(3)


def test_kernels_launched_early_wait_first_and_read_coherently():
    launched, waiting = set(), {}
    for _, text in sources():
        launched |= set(re.findall(r"launch_pdl\((k_\w+)", text))
        for name, params, first in kernels(text):
            if re.match(r"\s*pdl_\w+\([\w.]*\)\s*;", first):
                waiting[name] = params
    assert len(launched) > 15
    assert launched <= set(waiting), sorted(launched - set(waiting))
    for name, params in waiting.items():
        assert "__restrict__" not in params, name

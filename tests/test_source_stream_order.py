"""Source check: every fill the library issues names a stream.

The context's stream does not wait for the default stream, so a ``cudaMemset`` there may land after the
kernels that rely on it (a reduction's ticket, a solver's scratch)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluxion_b200", "csrc")


def test_no_memset_on_the_default_stream():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            for i, line in enumerate(f, 1):
                if re.search(r"\bcudaMemset\s*\(", line):
                    found.append(f"{os.path.basename(path)}:{i}")
    assert not found, found


def test_fills_name_the_contexts_stream():
    """cudaMemsetAsync with its fourth argument left out is the default stream too."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            src = f.read()
        for m in re.finditer(r"\bcudaMemsetAsync\s*\(", src):
            depth, k, commas = 1, m.end(), 0
            while depth:
                depth += {"(": 1, ")": -1}.get(src[k], 0)
                commas += src[k] == "," and depth == 1
                k += 1
            if commas != 3:
                found.append(f"{os.path.basename(path)}: {src[m.start():k]}")
    assert not found, found

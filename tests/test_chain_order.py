"""Chained tensor-core kernels (programmatic dependent launch) let the next
kernel's CTAs in only once their own tensor memory is allocated: otherwise a
successor's CTA beside a CTA that has released but not yet allocated could take
the SM's tensor memory and wait for the CTA that waits for it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "flowmc_gb300" / "csrc"


def _bodies(text):
    """(name, body) of every __global__ function of a source file, comments dropped."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        start = text.index("{", text.index(")", text.index("err)", m.end()) if "err)" in text[m.end():] else m.end()))
        depth, i = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield re.findall(r"(k_\w+)\s*\(", text[m.end():start])[0], text[start:i]


def _chained():
    found = []
    for f in sorted(CSRC.glob("tc_*.cu*")):
        found += [(f.name, n, b) for n, b in _bodies(f.read_text()) if "chain_release" in b or "chain_wait" in b]
    return found


def test_every_chained_kernel_is_seen():
    assert {n for _, n, _ in _chained()} == {"k_tc_gemm", "k_tc_spline", "k_tc_spline_bwd"}


@pytest.mark.parametrize("file,name,body", _chained(), ids=lambda v: v if isinstance(v, str) and len(v) < 40 else "")
def test_release_follows_the_allocation(file, name, body):
    releases = [m.start() for m in re.finditer(r"chain_release\(\)", body)]
    allocs = [m.start() for m in re.finditer(r"tcgen05\.alloc|pipe_setup<", body)]
    waits = [m.start() for m in re.finditer(r"chain_wait\(\)", body)]
    assert len(releases) == 1 and allocs
    assert max(allocs) < releases[0] < max(waits)
    assert body.count("__syncthreads", max(allocs), releases[0]) + body.count("pipe_setup<") > 0   # all warps are past it
    # the path of a launch that does no work waits too
    skip = body.index("tc_skip")
    assert skip < min(waits) < body.index("return;", skip)

"""The build's staleness check sees every header a source includes."""
import re

from flowmc_gb300 import build


def test_every_included_header_is_watched():
    watched = {h.name for h in build._headers()}
    included = set()
    for src in list(build.CSRC.iterdir()) + list(build.INCLUDE.iterdir()):
        if src.suffix in (".cu", ".cuh", ".h"):
            included |= {i.rsplit("/", 1)[-1] for i in re.findall(r'#include "([^"]+)"', src.read_text())}
    assert included and included <= watched, included - watched

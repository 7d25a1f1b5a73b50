"""The build compiles anew when a header that a source includes is newer, those of the kernels included."""
import os
import re

from porousmediaanalysis_gb300 import build


def test_headers_are_watched():
    watched = {os.path.basename(h) for h in build._headers()}
    for src in os.listdir(build.CSRC):
        with open(os.path.join(build.CSRC, src)) as f:
            included = {os.path.basename(i) for i in re.findall(r'#include "([^"]+)"', f.read())}
        assert included <= watched, (src, included - watched)

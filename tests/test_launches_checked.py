"""Every kernel launched with <<< >>> is followed by a look at the runtime's error record before
anything that may clear it: the launch helpers and the occupancy queries, which do."""

import os
import re

import pytest

from materialite_b200.csrc import build

CLEARING = re.compile(r"\bCKR\(|\blaunch_\w+(<[^;]*?>)?\(|persistent_grid\(|apply_projection_dev|cudaStreamEndCapture|\n}")


@pytest.mark.parametrize("name", sorted(os.path.basename(s) for s in build.sources()))
def test_plain_launches_are_checked(name):
    text = open(os.path.join(build.HERE, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"(\w+)(<[^<>;]*>)?\s*<<<", text):
        end = text.index(";", text.index(">>>", m.end()))
        rest = text[end:]
        checked, cleared = rest.find("cudaGetLastError()"), CLEARING.search(rest)
        assert checked >= 0 and (cleared is None or checked < cleared.start()), m.group(1)

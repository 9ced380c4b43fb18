"""Every kernel launch of the library is followed, in its own function, by a
check of the launch error: an unchecked one surfaces at some later call, after
results that were never written have been handed out."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pagani-toolkit_b200", "csrc")


@pytest.mark.parametrize("name", sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu"))))
def test_launches_are_checked(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    unchecked = []
    for m in re.finditer(r"<<<", text):
        end = text.find("\n}", m.start())
        if not re.search(r"PG_LAUNCHED\(|cudaGetLastError\(", text[m.start():end]):
            unchecked.append(text[:m.start()].count("\n") + 1)
    assert not unchecked, f"{name}: launches without a check at lines {unchecked}"

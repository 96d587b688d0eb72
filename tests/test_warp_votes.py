"""Warp votes and shuffles name the lanes that take part: the mask of the lanes that happen to be converged is not one that
a result may depend on."""
import os
import re

from conftest import PKG_NAME, ROOT


def test_no_vote_over_the_converged_lanes():
    csrc = os.path.join(ROOT, PKG_NAME, "csrc")
    for name in sorted(os.listdir(csrc)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, name)).read())
        assert "__activemask" not in text, name

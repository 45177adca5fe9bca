"""Warp votes name their lanes: by a mask known to all of them, or by a cooperative group, which is
formed and asked as one. A mask from __activemask() says only which lanes happened to be together
when it was read; lanes that it names and that do not come leave the others waiting."""
import os
import re

from yune_gb300 import build


def test_no_vote_over_the_lanes_that_happen_to_be_active():
    found = []
    for d, _, names in os.walk(build.CSRC):
        for n in names:
            text = re.sub(r"//[^\n]*", "", open(os.path.join(d, n)).read())
            found += [n] * ("__activemask" in text)
    assert not found

"""A shared array that is cleared as wider words than its elements declares their
alignment."""
import glob
import os
import re

import pytest

from conftest import PKG


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu"))),
                         ids=os.path.basename)
def test_widened_shared_arrays_are_aligned(path):
    src = open(path).read()
    for name in set(re.findall(r"reinterpret_cast<uint32_t\*>\((\w+)\)", src)):
        for decl in re.findall(rf"__shared__[^;]*\b(?:uint16_t|uint8_t|char)\s+{name}\[[^;]*;", src):
            assert "__align__(4)" in decl, decl

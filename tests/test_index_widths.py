"""A kernel that has a thread for each of several words an atom counts its threads
in 64 bits: three words an atom pass 2^31 from 715,827,883 atoms on."""
import glob
import os
import re

import pytest

from conftest import PKG


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu"))),
                         ids=os.path.basename)
def test_thread_index_holds_words_per_atom(path):
    src = open(path).read()
    narrow = re.findall(r"int32_t (\w+) = (?:\(int32_t\))?\(?blockIdx\.x \* blockDim\.x \+ threadIdx\.x"
                        r"\)?;\s*if \(\1 (?:<|>=) (\d+ \* n)\b", src)
    assert narrow == [], narrow

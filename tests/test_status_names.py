"""Every status bit of the library has a name in the Python layer.  CPU only."""
import os
import re

from abd_warp_b200 import _lib

SRC = os.path.join(os.path.dirname(os.path.abspath(_lib.__file__)), "csrc", "abd_common.cuh")


def test_every_bit_has_a_name():
    bits = {int(v) for v in re.findall(r"\bST_[A-Z_]+ = (\d+),", open(SRC).read())}
    assert len(bits) > 10 and bits == set(_lib.STATUS_NAMES)
    assert len(set(_lib.STATUS_NAMES.values())) == len(bits)

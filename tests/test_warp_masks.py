"""Warp votes, shuffles and synchronisations name the lanes that take part.
The lanes that happen to be active together (__activemask) are the compiler's
choice, so a value that depends on them can change with the next build."""
import re

import pytest

from tdycore_gb300.build import CSRC

SOURCES = sorted(p.name for p in CSRC.iterdir() if p.suffix in (".cu", ".h"))


@pytest.mark.parametrize("name", SOURCES)
def test_masks_are_defined(name):
    code = re.sub(r"//.*", "", (CSRC / name).read_text())
    assert not re.search(r"__activemask|__(any|all|ballot|shfl(_up|_down|_xor)?)\(|\bactivemask\b", code)

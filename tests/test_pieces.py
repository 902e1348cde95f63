"""16-byte accesses of complex rows. A complex number of the kernels (cpx) is aligned to its element, 4 or 8 bytes, so an
array of them that is kept in memory may start off a 16-byte boundary; the rows that are moved 16 bytes at a time have the
alignment in their type (cpx_row, checked by the compiler), and nothing else is viewed as such pieces."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'mom25d_b200', 'csrc')
VIEW = re.compile(r'reinterpret_cast<\s*(?:const\s+)?u?int4\s*\*\s*>')


def test_pieces_only_of_aligned_rows():
    found = {}
    for f in sorted(os.listdir(CSRC)):
        src = open(os.path.join(CSRC, f)).read()
        if f == 'common.cuh':                              # the one place: inside cpx_row
            i = src.find('struct __align__(16) cpx_row')
            src = src if i < 0 else src[:i] + src[src.index('\n};', i):]
        if VIEW.search(src):
            found[f] = len(VIEW.findall(src))
    assert not found, found

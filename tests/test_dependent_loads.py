"""Kernels that start while their predecessor drains read its results with plain loads.

ld.global.nc (__ldg) is defined only for memory that nothing writes during the kernel's
lifetime.  A kernel launched by launch_after() may be resident while the kernel before it
still writes, so no read-only load may name what the kernels of an extraction write: the
sign words, the masks of active words, the piece counts, the tiles' sums, the vertex
prefixes and the totals.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'meshing.jl_gb300', 'csrc')
WRITTEN = ('bits', 'wmask', 'pc', 'tsum', 'vpre', 'totals', 'work', 'done', 'vol_off')


def test_no_read_only_load_of_what_the_chain_writes():
    for name in ('k_bits.cu', 'k_emit_bits.cu', 'k_emit_shared.cu'):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        assert 'after_previous();' in text
        # the written arrays, and local pointers into them
        names = set()
        for m in re.finditer(r'\*\s*(\w+)\s*=\s*[^;]*?(?:p|v|P)\.(\w+)\b', text):
            if m.group(2) in WRITTEN:
                names.add(m.group(1))
        for m in re.finditer(r'(?:__ldg|ldv)\(([^()]*)', text):
            arg = m.group(1)
            assert not re.search(r'\b[pvP](?:\.|->)(?:%s)\b' % '|'.join(WRITTEN), arg), (name, m.group(0))
            assert arg.split('+')[0].strip(' &*') not in names, (name, m.group(0))

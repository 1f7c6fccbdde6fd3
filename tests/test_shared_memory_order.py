"""Shared memory that one thread writes and another one reads needs a CTA barrier
in between; where a missing one would show only once in many runs, the order in
the source is checked."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'bolt_b200', 'csrc')


def _source(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r'//[^\n]*', '', src)


def test_currents_are_zeroed_before_a_barrier():
    """The q-stage tile kernel's current sums: zeroed by index, added to by tile
    row and column.  The prologue that stands between ends in a barrier that
    every thread reaches."""
    src = _source('qpair_kernel.cuh')
    kernel = src[src.index('qpair_kernel(const __grid_constant__'):]
    zero = re.search(r'jacc\[c\]\s*=\s*0\.0', kernel).start()
    add = re.search(r'jacc\[[^\]]*\]\s*\+=|add_currents\(j', kernel).start()
    call = kernel.index('qpair_prologue<')
    assert zero < call < add
    prologue = src[src.index('void qpair_prologue('):]
    body = prologue[:re.search(r'\n}', prologue).start()]
    assert body.rstrip().endswith('__syncthreads();')

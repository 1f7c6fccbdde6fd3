"""Barriers whose absence or misuse would show only once in many runs, if ever: the
source is checked for them.  Shared memory that one thread writes and another one
reads needs a CTA barrier in between, and a barrier of the .aligned form needs a
converged warp."""

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


def test_cluster_barrier_takes_diverged_warps():
    """Between the passes of the field update, whose loops the threads of a warp leave
    at different times."""
    src = _source('fdtd_kernels.cuh')
    barrier = src[src.index('void cluster_barrier()'):]
    barrier = barrier[:barrier.index('}')]
    assert 'barrier.cluster.arrive.release;' in barrier
    assert 'barrier.cluster.wait.acquire;' in barrier
    assert '.aligned' not in barrier


def test_dynamic_shared_memory_has_one_alignment():
    """The kernels of a translation unit share the declaration: TMA's destinations in
    one of them need the 128 bytes that another one must not take back."""
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(('.cuh', '.cu', '.h')):
            found += re.findall(r'extern\s+__shared__\s+__align__\((\d+)\)[^;]*;', _source(name))
    assert len(found) >= 4 and set(found) == {'128'}

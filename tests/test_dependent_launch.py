"""Rules of kernels launched as programmatic dependents, read from the sources
(what breaks one would be a hang or a stale value on the GPU):

* tensor memory is allocated, and the block has met at a barrier since, before
  the kernel lets its dependents start: else a dependent's block on the same SM
  may take the columns that a block it waits for still needs."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(
    __file__))), 'quantumsim_gb300', 'csrc')


def kernels():
    """(file, name, parameters, body without comments) of every __global__."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, '*.cu'))):
        with open(path) as f:
            text = re.sub(r'//[^\n]*', '', f.read())
        for m in re.finditer(r'__global__\s+void\b', text):
            b = text.index('{', m.end())
            depth, e = 1, b + 1
            while depth:
                depth += {'{': 1, '}': -1}.get(text[e], 0)
                e += 1
            head = text[m.end():b]
            # the name stands before the parameter list, the last parentheses
            name = re.search(r'(\w+)\s*\((?:[^()]|\([^()]*\))*\)\s*$', head)
            out.append((os.path.basename(path), name.group(1), head,
                        text[b:e]))
    return out


DEPENDENT = [k for k in kernels() if 'pdl_wait()' in k[3]]


def test_some_are_found():
    names = {k[1] for k in DEPENDENT}
    assert {'gather_kernel', 'grad_stage2', 'apply_ptm_kernel',
            'apply16_umma_kernel', 'apply_wide_kernel'} <= names


@pytest.mark.parametrize('k', DEPENDENT, ids=lambda k: k[1])
def test_tensor_memory_before_dependents(k):
    body = k[3]
    before = body[:body.index('pdl_wait()')]
    if 'tcgen05.alloc' not in body:
        return
    alloc = before.rindex('tcgen05.alloc')  # before the wait
    assert '__syncthreads()' in before[alloc:]

"""Rules of kernels launched as programmatic dependents, read from the sources
(what breaks one would be a hang or a stale value on the GPU):

* tensor memory is allocated, and the block has met at a barrier since, before
  the kernel lets its dependents start: else a dependent's block on the same SM
  may take the columns that a block it waits for still needs;
* what a kernel reads is not read-only while it runs (its predecessor may still
  be writing it), so no pointer to const memory is __restrict__."""
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
        if path.endswith('qsgb_jit.cu'):
            continue  # text of generated kernels: below
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


READ_ONLY = re.compile(r'const\s+[\w:]+\s*\*\s*(?:const\s+)?__restrict__')


@pytest.mark.parametrize('k', DEPENDENT, ids=lambda k: k[1])
def test_nothing_read_is_declared_read_only(k):
    assert not READ_ONLY.search(k[2] + k[3])


@pytest.mark.parametrize('path', sorted(glob.glob(os.path.join(CSRC, '*.cu'))),
                         ids=os.path.basename)
def test_nor_in_the_functions_they_call(path):
    here = [k for k in kernels() if k[0] == os.path.basename(path)]
    if not here or any(k not in DEPENDENT for k in here):
        return  # files whose kernels are all launched so
    with open(path) as f:
        assert not READ_ONLY.search(re.sub(r'//[^\n]*', '', f.read()))


def test_generated_kernels_pass_their_pointer_through_the_wait():
    """They keep __restrict__ (loads move above stores) on a pointer that comes
    out of an asm behind the wait."""
    with open(os.path.join(CSRC, 'qsgb_jit.cu')) as f:
        text = f.read()
    waits = [m.end() for m in re.finditer(r'qsgb_pdl_wait\(\);', text)]
    assert len(waits) == text.count('"extern \\"C\\" __global__') + 1 == 3
    # the vector loads of a group stay behind the wait as volatile asm
    loads = re.findall(r'asm(?: volatile)?\(\\"ld\.global', text)
    assert len(loads) == 2 and all('volatile' in x for x in loads)
    for w in waits:
        assert text[w:].startswith(
            '\\n  asm volatile(\\"\\" : \\"+l\\"(in));')

"""The term limit of the run-time specialised kernels is one number: the
library's, the per-call path's and the planner's."""
import os
import re

from quantumsim_gb300 import build, circuit, ops


def test_one_limit():
    with open(os.path.join(build.CSRC, 'qsgb_jit.h')) as f:
        (n,) = re.findall(r'kMaxJitTerms = (\d+);', f.read())
    assert int(n) == ops.MAX_JIT_TERMS == circuit.MAX_SPECIALISED_TERMS

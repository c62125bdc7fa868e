"""The default split of a batched step: its dP partials are bounded by the
device's blocks, not by the number of instances."""
import numpy as np
import pytest

from quantumsim_gb300 import batch as BT

GRID = 304


def _program(ns, depth, tile):
    specs = [BT.CircuitSpec(n, depth, i) for i, n in enumerate(ns)]
    units = [BT.plan_units(s.ops()) for s in specs]
    base = np.cumsum([0] + [len(u) for u in units])
    return BT.build_program(units, base, [4 ** n for n in ns],
                            [depth] * len(ns), 8, tile, grid=GRID)


@pytest.mark.parametrize('ns', [[10] * 64, [10] * 256, [8] * 512, [12] * 20,
                                [4, 6, 8, 10] * 40, [14] * 4])
def test_items_per_stage(ns):
    items, begin, n_slots = _program(ns, 6, 0)
    per_stage = np.diff(begin)[:-1]
    # the last item of an entry may be a part of one
    assert per_stage.max() <= BT.ADAPT_ITEMS * GRID + len(ns)
    adjoint = int((items['op'] == BT.BOP_ADJOINT).sum())
    assert n_slots == adjoint
    stages = len({int(s) for s in np.flatnonzero([
        (items['op'][begin[s]:begin[s + 1]] == BT.BOP_ADJOINT).any()
        for s in range(len(begin) - 2)])})
    assert n_slots * 2048 <= stages * (BT.ADAPT_ITEMS * GRID + len(ns)) * 2048


def test_many_instances_take_no_more_than_fixed_tiles():
    ns = [10] * 512
    assert _program(ns, 6, 0)[2] <= _program(ns, 6, 8192)[2]

"""Items sized per stage (tile 0): every entry's items cover its range exactly
once in steps the kernel accepts, no stage leaves most blocks idle while it
has work for them, and on the GPU the results are those of fixed tiles."""
import numpy as np
import pytest

from quantumsim_gb300 import batch as BT


def _program(ns, depth, grid):
    specs = [BT.CircuitSpec(n, depth, i) for i, n in enumerate(ns)]
    units = [BT.plan_units(s.ops()) for s in specs]
    base = np.cumsum([0] + [len(u) for u in units])
    return BT.build_program(units, base, [4 ** n for n in ns],
                            [depth] * len(ns), 8, 0, grid=grid)


@pytest.mark.parametrize('grid', [1, 304])
@pytest.mark.parametrize('ns', [[1], [2, 3], [8] * 5, [4, 9, 12], [12] * 7,
                                [5, 6, 11] * 6])
def test_items_cover_ranges(ns, grid):
    items, begin, n_slots = _program(ns, 10, grid)
    slots = []
    for s in range(len(begin) - 2):
        st = items[begin[s]:begin[s + 1]]
        elems = 0
        for key in {(int(i['inst']), int(i['op']), int(i['ptm']),
                     int(i['q0'])) for i in st}:
            mine = np.sort(st[(st['inst'] == key[0]) & (st['op'] == key[1]) &
                              (st['ptm'] == key[2]) & (st['q0'] == key[3])],
                           order='beg')
            width = {BT.BOP_APPLY: 16, BT.BOP_ADJOINT: 16}.get(key[1], 1)
            if width == 16 and mine[0]['q1'] < 0:
                width = 4
            total = 1 if key[1] == BT.BOP_LOSS else 4 ** ns[key[0]] // width
            if key[1] != BT.BOP_LOSS:
                assert mine[0]['beg'] == 0 and mine[-1]['end'] == total
                assert np.all(mine['end'][:-1] == mine['beg'][1:])
                assert np.all(mine['beg'] % 4 == 0)
                assert np.all(mine['end'] > mine['beg'])
                elems += total * width
            if width > 1:  # folds of the FP32 gradient sums stay whole
                assert np.all(mine['beg'] * width % BT.ADAPT_STEP == 0)
            if key[1] == BT.BOP_ADJOINT:
                slots += list(mine['slot'])
        # every block has its share of a large stage, and none too many items
        if elems >= 2 * grid * BT.ADAPT_STEP:
            assert len(st) >= 0.5 * grid
        assert len(st) <= (BT.ADAPT_ROUNDS + 1) * grid + 65 * len(ns)
    assert sorted(slots) == list(range(n_slots))


@pytest.mark.gpu
@pytest.mark.parametrize('ns', [[1, 2, 3], [7, 4, 9], [10, 10]])
def test_results_match_fixed_tiles(ns):
    import torch
    specs = [BT.CircuitSpec(n, 9, 5 + i) for i, n in enumerate(ns)]
    rng = np.random.default_rng(1)
    targets = []
    for n in ns:
        t = rng.exponential(size=2 ** n) + 1e-3
        targets.append(torch.from_numpy(t / t.sum()))
    got = []
    for tile in (None, 2048):
        sim = BT.BatchedSimulator(specs, targets, tile=tile)
        if tile is None:
            sim._build_program(0)  # whatever tile is cached on this machine
        sim.set_ptms([BT.instance_ptms(s) for s in specs])
        sim.step()
        sim.check()
        got.append((sim.prob.clone(), sim.loss.clone(), sim.op_grad.clone()))
    assert torch.equal(got[0][0], got[1][0])
    assert torch.allclose(got[0][1], got[1][1], rtol=1e-12, atol=0)
    # the same FP32 sums, added in FP64 in another order
    scale = got[1][2].abs().max()
    assert float((got[0][2] - got[1][2]).abs().max()) <= 1e-13 * float(scale)

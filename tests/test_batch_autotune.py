"""autotune times the default split too, and what it finds is what a later
simulator of the same circuits takes: a stored 0 is a choice, an entry written
before the default split was among the candidates is not."""
import inspect
import json

import pytest

from quantumsim_gb300 import batch as BT


class _Sim(BT.BatchedSimulator):
    def __init__(self):
        self.specs = [BT.CircuitSpec(n, 2, n) for n in (3, 5)]
        self.max_grid, self.n_ptm = 304, 17


@pytest.fixture
def cache(tmp_path, monkeypatch):
    path = tmp_path / 'tiles.json'
    monkeypatch.setenv('QSGB_AUTOTUNE_CACHE', str(path))
    return path


def test_default_split_is_a_candidate():
    default = inspect.signature(
        BT.BatchedSimulator.autotune).parameters['candidates'].default
    assert default[0] == 0


def test_stored_choices(cache):
    sim = _Sim()
    assert sim._cached_tile() is None
    cache.write_text(json.dumps({sim._cache_key(): {'tile': 0}}))
    assert sim._cached_tile() == 0
    # the key as it was before
    cache.write_text(json.dumps(
        {'2:{}:304:17'.format(4 ** 3 + 4 ** 5): {'tile': 2048}}))
    assert sim._cached_tile() is None


@pytest.mark.gpu
def test_choice_is_reloaded(cache):
    import torch
    specs = [BT.CircuitSpec(n, 3, n) for n in (3, 5, 6)]
    targets = [torch.full((2 ** s.n,), 2.0 ** -s.n, dtype=torch.float64)
               for s in specs]

    def make(**kw):
        sim = BT.BatchedSimulator(specs, targets, **kw)
        sim.set_ptms([BT.instance_ptms(s) for s in specs])
        return sim

    sim = make()
    assert sim.tile == 0
    times = sim.autotune(reps=1)
    assert 0 in times and len(times) == 6
    assert sim.autotune(candidates=(64,), reps=1).keys() == {64}
    assert make().tile == 64          # a fixed tile was the last one found
    assert make(tile=0).tile == 0     # but a caller's choice stands
    assert sim.autotune(candidates=(0,), reps=1).keys() == {0}
    assert make().tile == 0 and make(tile=32).tile == 32

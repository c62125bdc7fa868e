"""Two-qubit adjoint of the batched step: items that start at any multiple of
4 groups and end inside a tile, targets at every distance from the last qubit,
against FP64 gradients of the plain path."""
import pytest
import torch

from quantumsim_gb300 import batch as BT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('tile', (0, 4, 12, 36, 40))
def test_items_at_any_offset(tile):
    specs = [BT.CircuitSpec(n, 8, 40 + n) for n in (2, 3, 4, 5, 6, 7)]
    targets = [BT.target_probabilities(s, 7 + i) for i, s in enumerate(specs)]
    ptms = [BT.instance_ptms(s) for s in specs]
    sim = BT.BatchedSimulator(specs, targets, checkpoint_every=4)
    sim._build_program(tile, max_items=1 << 20)
    sim.set_ptms(ptms)
    sim.step(use_graph=False)
    torch.cuda.synchronize()
    sim.check()
    probs, _, grads = sim.results()
    for s, p, t, pr, gr in zip(specs, ptms, targets, probs, grads):
        p64, _, g64 = BT.plain_gradients(s, p, t, dtype=torch.float64,
                                         checkpoint_every=4)
        assert float((pr - p64).abs().max()) < 1e-6
        # FP32 states (2^-24) through some 50 ops and 1 / p of the loss: as
        # the comparison of whole steps
        scale = max(float(g.abs().max()) for g in g64)
        for a, b in zip(gr, g64):
            assert float((a - b.to(a.device)).abs().max()) < 1e-4 * scale

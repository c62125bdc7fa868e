"""Workloads for measuring the GB300 density-matrix backend.

Each case is what a user of the package runs, through its public entry
points: circuits applied unit by unit, fused or as a captured graph, the
readout of a state, differentiated layers, a graph-replayed gradient step and
a batch of circuits.  ``listed()`` gives the fixed cases, ``draw(rng)`` one
more of the same ranges.  A case holds its sizes and the seed of its
structure (which gates act where); ``prepare(case, seed)`` draws the values
(the state, angles, noise rates, targets) from `seed` alone.

``exact(case, seed)`` evaluates the same inputs in float64 with plain torch.
"""
import functools
import math

import numpy as np
import torch

import quantumsim_gb300 as qg
from quantumsim_gb300 import bases, batch, fitting, ptm as P

T_1Q = 20e-9
T_2Q = 40e-9


def listed():
    return [
        # a small circuit simulated gate by gate, as a quantumsim operation
        # chain does: 180 calls whose latency is all that counts
        {'name': 'units_6q', 'kind': 'units', 'n': 6, 'layers': 20,
         'dtype': 'f64', 'circuit': 0},
        # the same kind of circuit planned once and replayed for many inputs
        {'name': 'graph_7q', 'kind': 'graph', 'n': 7, 'layers': 20,
         'dtype': 'f64', 'circuit': 1},
        # what is read from a state after a circuit, then a projective
        # measurement of one qubit
        {'name': 'readout_12q', 'kind': 'readout', 'n': 12, 'dtype': 'f64',
         'circuit': 2},
        # one layer of a large noisy circuit, unit by unit (the benchmark's
        # size): rotations on every qubit, CZs on random ordered pairs
        {'name': 'noisy_14q', 'kind': 'noisy', 'n': 14, 'layers': 1,
         'dtype': 'f64', 'circuit': 3},
        # the same in the FP32 storage option, on an odd number of qubits
        {'name': 'noisy_13q_f32', 'kind': 'noisy', 'n': 13, 'layers': 1,
         'dtype': 'f32', 'circuit': 4},
        # random two-qubit unitaries with damping on random pairs (a layer of
        # a quantum-volume circuit): dense 16 x 16 PTMs
        {'name': 'dense_12q', 'kind': 'dense', 'n': 12, 'layers': 1,
         'dtype': 'f64', 'circuit': 5},
        # leakage simulation on qutrits: 9 x 9 gates, 81 x 81 CZs, and a
        # mid-circuit measurement with its basis reduction
        {'name': 'qutrits_8', 'kind': 'qutrits', 'n': 8, 'layers': 1,
         'dtype': 'f64', 'circuit': 6},
        # general two-qutrit gates: dense 81 x 81 PTMs
        {'name': 'qutrits_dense_7', 'kind': 'qutrits_dense', 'n': 7,
         'layers': 1, 'dtype': 'f64', 'circuit': 7},
        # a noisy circuit through the fused executor and the partial trace of
        # its result
        {'name': 'fused_13q', 'kind': 'fused', 'n': 13, 'layers': 8,
         'dtype': 'f64', 'circuit': 8},
        # one layer forward and backward through autograd: the gradients of
        # the state and of every PTM
        {'name': 'diff_11q', 'kind': 'diff', 'n': 11, 'layers': 1,
         'dtype': 'f64', 'ptms': 'host', 'circuit': 9},
        # one gradient step of the 249-parameter noise model
        {'name': 'grad_step_10q', 'kind': 'grad', 'n': 10, 'layers': 40,
         'groups': 22, 'dtype': 'f64', 'circuit': 3},
        # one gradient step of many uneven circuits in one launch (FP32)
        {'name': 'batch_20', 'kind': 'batch', 'count': 20, 'n_min': 4,
         'n_max': 12, 'layers': 30, 'circuit': 10},
    ]


def draw(rng):
    kind = rng.choice(('units', 'graph', 'readout', 'noisy', 'dense',
                       'qutrits', 'qutrits_dense', 'fused', 'diff', 'grad',
                       'batch'))
    c = {'kind': kind, 'circuit': rng.randrange(100, 1000000)}
    dtype = rng.choice(('f64', 'f64', 'f32'))
    if kind in ('units', 'graph'):
        c.update(n=rng.randint(3, 9), layers=rng.randint(4, 20), dtype=dtype)
    elif kind == 'readout':
        c.update(n=rng.randint(3, 14), dtype=dtype)
    elif kind == 'noisy':
        c.update(n=rng.randint(10, 14), layers=rng.randint(1, 2), dtype=dtype)
    elif kind == 'dense':
        c.update(n=rng.randint(4, 14), layers=rng.randint(1, 2), dtype=dtype)
    elif kind == 'qutrits':
        c.update(n=rng.randint(3, 8), layers=rng.randint(1, 2), dtype=dtype)
    elif kind == 'qutrits_dense':
        c.update(n=rng.randint(2, 8), layers=1, dtype=dtype)
    elif kind == 'fused':
        c.update(n=rng.randint(8, 13), layers=rng.randint(3, 8), dtype=dtype)
    elif kind == 'diff':
        c.update(n=rng.randint(4, 12), layers=rng.randint(1, 2), dtype=dtype,
                 ptms=rng.choice(('host', 'device')))
    elif kind == 'grad':
        c.update(n=rng.randint(4, 10), layers=rng.randint(8, 40),
                 groups=rng.randint(2, 8), dtype=dtype)
    else:
        c.update(count=rng.randint(4, 20), n_min=rng.randint(3, 5),
                 n_max=rng.randint(8, 12), layers=rng.randint(10, 30))
    return c


# ---------------------------------------------------------------- inputs
def _dtype(case):
    return torch.float32 if case.get('dtype') == 'f32' else torch.float64


def _state(n, d, seed, dtype):
    """A mixed, correlated state: the weighted sum of three products of
    random one-qudit density matrices, as a Pauli vector on the GPU."""
    rng = np.random.default_rng([seed, 1])
    vec = np.asarray(bases.general(d).vectors)
    out = None
    for weight in (0.5, 0.3, 0.2):
        x = torch.full((1,), weight, dtype=torch.float64, device='cuda')
        for _ in range(n):
            a = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
            rho = a @ a.conj().T
            rho /= np.trace(rho).real
            v = np.einsum('xij,ji->x', vec, rho).real
            x = torch.outer(x, torch.from_numpy(v).cuda()).reshape(-1)
        out = x if out is None else out.add_(x)
    return out.to(dtype).reshape((d * d,) * n)


def _times(rng, n):
    t1 = rng.uniform(20e-6, 60e-6, n)
    return t1, rng.uniform(10e-6, t1)


def _unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) +
                        1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _random_pairs(rng, n, count):
    return [tuple(int(q) for q in rng.choice(n, 2, replace=False))
            for _ in range(count)]


def _line_pairs(rng, n, layer):
    return [(i, i + 1) if rng.integers(2) else (i + 1, i)
            for i in range(layer % 2, n - 1, 2)]


def _gates(case, seed):
    """[(ptm, qudits)] of the case's circuit, float64 numpy PTMs."""
    kind, n = case['kind'], case['n']
    s = np.random.default_rng([case['circuit'], 2])  # structure
    v = np.random.default_rng([seed, 3])             # values
    out = []
    t1, t2 = _times(v, n)
    b3 = bases.general(3)
    for layer in range(case['layers']):
        if kind == 'dense':
            for a, b in _random_pairs(s, n, n // 2):
                damp = P.kron(*(P.amp_phase_damping(*P.damping_rates(
                    t1[q], t2[q], T_2Q)) for q in (a, b)))
                gate = P.kraus_to_ptm(_unitary(v, 4), (bases.general(2),) * 2)
                out.append((P.compose(gate, damp).numpy(), (a, b)))
        elif kind == 'qutrits_dense':
            for pair in _line_pairs(s, n, layer):
                out.append((P.kraus_to_ptm(_unitary(v, 9), (b3, b3)).numpy(),
                            pair))
        elif kind == 'qutrits':
            for q in range(n):
                rot = P.rotate('xy'[s.integers(2)],
                               v.uniform(0, 2 * math.pi), b3)
                damp = v.uniform(2e-4, 1e-3)
                noise = P.qutrit_amp_damping(0.0, v.uniform(1e-4, 1e-2), damp,
                                             2 * damp, b3)
                out.append((P.compose(rot, noise).numpy(), (q,)))
            for pair in _line_pairs(s, n, layer):
                out.append((P.qutrit_cphase(
                    math.pi + v.normal(0, 0.02),
                    v.uniform(1e-4, 1e-2)).numpy(), pair))
        else:
            for q in range(n):
                out.append((P.noisy_rotation(
                    'xyz'[s.integers(3)], v.uniform(0, 2 * math.pi), t1[q],
                    t2[q], T_1Q).numpy(), (q,)))
            pairs = _line_pairs(s, n, layer) \
                if kind in ('units', 'graph', 'diff') \
                else _random_pairs(s, n, n // 2)
            for a, b in pairs:
                out.append((P.noisy_cphase(math.pi, t1[a], t2[a], t1[b],
                                           t2[b], T_2Q).numpy(), (a, b)))
    return out


def _choice(case, count):
    """`count` distinct seeded qudits of the case, ascending."""
    rng = np.random.default_rng([case['circuit'], 4])
    return tuple(sorted(int(q) for q in
                        rng.choice(case['n'], count, replace=False)))


def _pauli_string(case):
    rng = np.random.default_rng([case['circuit'], 5])
    return ''.join('IXYZ'[i] for i in rng.integers(4, size=case['n']))


def _histogram(rng, size):
    """A measured distribution of a random circuit (exponentially
    distributed probabilities)."""
    t = rng.exponential(size=size) + 1e-3
    return torch.from_numpy(t / t.sum())


def _model(case, seed):
    model = fitting.NoisyCircuitModel(case['n'], case['layers'],
                                      case['groups'], seed=case['circuit'])
    target = _histogram(np.random.default_rng([seed, 6]), 2 ** case['n'])
    return model, target, model.perturbed(seed=seed)


def _batch(case, seed):
    s = np.random.default_rng([case['circuit'], 7])
    v = np.random.default_rng([seed, 8])
    ns = [int(n) for n in s.integers(case['n_min'], case['n_max'] + 1,
                                     case['count'])]
    ns[0] = case['n_max']
    specs = [batch.CircuitSpec(n, case['layers'], case['circuit'] + i)
             for i, n in enumerate(ns)]
    ptms = [batch.instance_ptms(sp, torch.from_numpy(
        v.normal(0, 0.5, (sp.depth, sp.n)))) for sp in specs]
    targets = [_histogram(v, 2 ** n) for n in ns]
    return specs, ptms, targets


def prepare(case, seed):
    kind = case['kind']
    st = {'case': case}
    if kind == 'grad':
        model, target, p = _model(case, seed)
        st['params'] = {k: t.cuda().requires_grad_(True)
                        for k, t in p.items()}
        st['step'] = fitting.GraphedGradient(model, target,
                                             dtype=_dtype(case))
        return st
    if kind == 'batch':
        specs, ptms, targets = _batch(case, seed)
        st['sim'] = batch.BatchedSimulator(specs, targets)
        st['sim'].set_ptms(ptms)
        return st
    n, d = case['n'], 3 if kind.startswith('qutrits') else 2
    st['bases'] = [bases.general(d)] * n
    st['x'] = _state(n, d, seed, _dtype(case))
    if kind == 'readout':
        st['keep'] = _choice(case, 2)
        st['string'] = _pauli_string(case)
        return st
    st['gates'] = _gates(case, seed)
    if kind == 'fused':
        st['circuit'] = qg.FusedCircuit(st['gates'])
        st['keep'] = _choice(case, 4)
    elif kind == 'graph':
        st['graph'] = qg.FusedCircuit(st['gates']).capture(_vector(st))
    elif kind == 'qutrits':
        st['measured'] = _choice(case, 1)[0]
    elif kind == 'diff':
        dev = 'cuda' if case['ptms'] == 'device' else 'cpu'
        st['x'].requires_grad_(True)
        st['ptms'] = [torch.from_numpy(p).to(dev).requires_grad_(True)
                      for p, _ in st['gates']]
        st['target'] = _histogram(np.random.default_rng([seed, 9]),
                                  2 ** n).cuda()
    return st


# ------------------------------------------------------------------ runs
def _vector(st):
    return qg.PauliVectorGB300(st['bases'], st['x'], force=True)


def run(st):
    kind = st['case']['kind']
    if kind == 'grad':
        for t in st['params'].values():
            t.grad = None
        loss = st['step'].step(st['params'])
        return {'loss': loss,
                'grads': {k: t.grad for k, t in st['params'].items()}}
    if kind == 'batch':
        sim = st['sim']
        sim.step()
        return {'prob': sim.prob, 'loss': sim.loss, 'grads': sim.op_grad}
    if kind == 'diff':
        y = st['x']
        for p, (_, qs) in zip(st['ptms'], st['gates']):
            y = qg.apply_ptm_diff(y, p, *qs)
        prob = qg.diagonal_diff(y, st['bases'])
        t = st['target']
        loss = torch.sum(t * (torch.log(t) - torch.log(prob)))
        grads = torch.autograd.grad(loss, [st['x']] + st['ptms'])
        return {'loss': loss, 'prob': prob, 'grads': grads}
    pv = _vector(st)
    if kind == 'readout':
        n = st['case']['n']
        out = {'trace': pv.trace(),
               'probs': [pv.meas_prob(q) for q in range(n)],
               'diagonal': pv.diagonal(),
               'reduced': pv.partial_trace(*st['keep']).to_pv(),
               'value': pv.exp_value(st['string'])}
        q = st['keep'][0]
        pv.project(q, int(out['probs'][q][1] > out['probs'][q][0]))
        out['weight'] = pv.renormalize()
        out['state'] = pv.data
        return out
    if kind == 'graph':
        return st['graph'].run(pv).data
    if kind == 'fused':
        st['circuit'](pv)
        return {'state': pv.data, 'reduced': pv.partial_trace(
            *st['keep']).to_pv()}
    for ptm, qs in st['gates']:
        pv.apply_ptm(ptm, *qs)
    if kind == 'units':
        return {'state': pv.data, 'diagonal': pv.diagonal()}
    if kind == 'qutrits':
        q = st['measured']
        b = pv.bases[q]
        probs = pv.meas_prob(q)
        pv.reduce_basis(q, [b.computational_basis_indices[i]
                            for i in range(3)])
        pv.project(q, int(np.argmax(probs)))
        return {'probs': probs, 'weight': pv.renormalize(),
                'state': pv.data}
    return pv.data


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: every application reads its input vector and writes its
    output.  Operations: the multiplications and additions of the PTMs'
    non-zero terms."""
    kind = case['kind']
    size = 4 if case.get('dtype') == 'f32' else 8
    if kind == 'batch':
        b = f = 0.0
        s = np.random.default_rng([case['circuit'], 7])
        ns = [int(n) for n in s.integers(case['n_min'], case['n_max'] + 1,
                                         case['count'])]
        ns[0] = case['n_max']
        for i, n in enumerate(ns):
            spec = batch.CircuitSpec(n, case['layers'], case['circuit'] + i)
            units = batch.plan_units(spec.ops())
            for _, qs, _ in units:
                # forward: read and write x; backward: read x and g, write
                # both (x rebuilt); three products of K terms each
                b += 24.0 * 4 ** n
                f += 4 * 2.0 * 4 ** n * 4 ** len(qs)
        return {'bytes': b, 'flops': f}
    n = case['n']
    if kind == 'grad':
        # per unit: forward, its recomputation, the state's gradient (read
        # and write) and the PTM's gradient (two reads)
        units = case['layers'] * ((n + 1) / 2.0)
        return {'bytes': units * 8 * size * 4.0 ** n,
                'flops': units * 4 * 2.0 * 16 * 4.0 ** n}
    if kind == 'readout':
        # the projection reads a quarter of the vector and the
        # renormalisation reads and writes it; diagonals are 2^n
        return {'bytes': size * 4.0 ** n + size * 2.0 ** n * (n + 2),
                'flops': 4.0 ** n / 4 + 2.0 ** n * (n + 2)}
    full = float((9 if kind.startswith('qutrits') else 4) ** n)
    one = 0 if 'dense' in kind else case['layers'] * n
    two = sum(n // 2 if kind not in ('units', 'graph', 'diff', 'qutrits',
                                     'qutrits_dense')
              else len(range(layer % 2, n - 1, 2))
              for layer in range(case['layers']))
    terms1, terms2 = {'dense': (0, 16), 'qutrits_dense': (0, 81),
                      'qutrits': (2.56, 2.14)}.get(kind, (2.5, 1.56))
    flops = 2 * full * (one * terms1 + two * terms2)
    passes = one + two
    if kind in ('fused', 'graph'):
        passes = two if n > 1 else one  # rotations merge into the CZs
    if kind == 'graph':
        passes = 1  # the vector is read and written once at the least
    b = passes * 2 * size * full
    if kind == 'diff':
        b += (one + two) * 4 * size * full  # g read and written, x and g read
        flops += 2 * full * (one * (2.5 + 4) + two * (1.56 + 16))
    return {'bytes': b, 'flops': flops}


# ----------------------------------------------------------------- exact
def _apply(x, p, qs):
    """P x on the axes `qs` of x, in float64."""
    k = len(qs)
    y = torch.tensordot(p, x, dims=(list(range(k, 2 * k)), list(qs)))
    return torch.movedim(y, list(range(k)), list(qs)).contiguous()


def _diag_index(n):
    """Position of the diagonal entries of n qubits (per qubit, the first
    two basis elements are the projectors on |0> and |1>)."""
    idx = torch.zeros(1, dtype=torch.long, device='cuda')
    for _ in range(n):
        idx = (idx[:, None] * 4 + torch.arange(2, device='cuda')).reshape(-1)
    return idx


def _loss(prob, t):
    return torch.sum(t * (torch.log(t) - torch.log(prob)))


def _exact_readout(case, x):
    n = case['n']
    keep, string = _choice(case, 2), _pauli_string(case)
    d = x.reshape(-1)[_diag_index(n)].reshape((2,) * n)
    probs = [d.sum(dim=[a for a in range(n) if a != q]) for q in range(n)]
    red = x
    for q in reversed(range(n)):
        if q not in keep:
            red = red.select(q, 0) + red.select(q, 1)
    r2 = math.sqrt(2.0)
    w = {'I': (1, 1, 0, 0), 'X': (0, 0, r2, 0), 'Y': (0, 0, 0, None),
         'Z': (1, -1, 0, 0)}
    # tr(Y b) of the fourth basis element, from its definition
    b3 = np.asarray(bases.general(2).vectors)[3]
    ey = float(np.trace(np.array([[0, -1j], [1j, 0]]) @ b3).real)
    val = x
    for ch in string:
        row = torch.tensor([ey if u is None else u for u in w[ch]],
                           dtype=torch.float64, device='cuda')
        val = torch.tensordot(row, val, dims=1)
    q = keep[0]
    k = int(probs[q][1] > probs[q][0])
    sub = x.narrow(q, k, 1).contiguous()
    tr = d.select(q, k).sum()
    return {'trace': float(d.sum()), 'probs': probs, 'diagonal': d.reshape(-1),
            'reduced': red, 'value': float(val), 'weight': float(tr),
            'state': sub / tr}


def _exact_grad(case, seed):
    model, target, p0 = _model(case, seed)
    n = model.n
    p = {k: t.cuda().requires_grad_(True) for k, t in p0.items()}
    groups = torch.arange(model.n_layers, device='cuda') % model.n_groups
    ang = model.base_angles.cuda() + p['angle_offset'][groups]
    c128 = torch.complex128
    vec = torch.from_numpy(np.asarray(bases.general(2).vectors)).cuda()
    vec2 = torch.einsum('aij,bkl->abikjl', vec, vec).reshape(16, 4, 4)

    def channel(kraus, v):
        return sum(torch.einsum('xij,...jl,ylm,...im->...xy', v, k, v,
                                k.conj()) for k in kraus).real

    def mat(rows):
        return torch.stack([torch.stack(r, -1) for r in rows], -2)

    c, s = torch.cos(ang / 2).to(c128), torch.sin(ang / 2).to(c128)
    z = torch.zeros_like(c)
    rots = {'x': [[c, -1j * s], [-1j * s, c]], 'y': [[c, -s], [s, c]],
            'z': [[c - 1j * s, z], [z, c + 1j * s]]}
    rots = {k: channel([mat(r)], vec) for k, r in rots.items()}
    t1, t2 = p['t1'] * 1e-6, p['t2'] * 1e-6
    gamma = 1 - torch.exp(-T_1Q / t1)
    lam = 1 - torch.exp(-2 * T_1Q * (1 / t2 - 1 / (2 * t1)))
    o, zz = torch.ones_like(t1), torch.zeros_like(t1)

    def damping(g, off):
        k0 = mat([[o, zz], [zz, torch.sqrt(1 - g)]]).to(c128)
        k1 = mat([[zz, torch.sqrt(g)], [zz, zz]] if off else
                 [[zz, zz], [zz, torch.sqrt(g)]]).to(c128)
        return channel([k0, k1], vec)
    damp = damping(lam, False) @ damping(gamma, True)
    ph = math.pi + p['cz_phase']
    cz = torch.diag_embed(torch.stack(
        [torch.ones_like(ph).to(c128)] * 3 + [torch.exp(1j * ph.to(c128))],
        -1))
    cz = channel([cz], vec2).reshape(-1, 4, 4, 4, 4)
    x = torch.zeros((4,) * n, dtype=torch.float64, device='cuda')
    x[(0,) * n] = 1
    for layer in range(model.n_layers):
        for q in range(n):
            x = _apply(x, damp[q] @ rots[model.axes[layer][q]][layer, q],
                       (q,))
        for i in range(layer % 2, n - 1, 2):
            x = _apply(x, cz[i], (i, i + 1))
    loss = _loss(x.reshape(-1)[_diag_index(n)], target.cuda())
    loss.backward()
    return {'loss': loss.detach(),
            'grads': {k: t.grad for k, t in p.items()}}


def _exact_batch(case, seed):
    specs, ptms, targets = _batch(case, seed)
    probs, losses = [], []
    grads = []
    for spec, ps, t in zip(specs, ptms, targets):
        n, t = spec.n, t.cuda()
        qs = [q for _, q in spec.ops()]
        ps = [p.cuda().reshape((4,) * (2 * len(q))) for p, q in zip(ps, qs)]
        x = torch.zeros((4,) * n, dtype=torch.float64, device='cuda')
        x[(0,) * n] = 1
        kept = []
        for p, q in zip(ps, qs):
            kept.append(x)
            x = _apply(x, p, q)
        idx = _diag_index(n)
        d = x.reshape(-1)[idx]
        probs.append(d)
        losses.append(_loss(d, t))
        g = torch.zeros(4 ** n, dtype=torch.float64, device='cuda')
        g[idx] = -t / d
        g = g.reshape((4,) * n)
        rows = []
        for p, q in zip(reversed(ps), reversed(qs)):
            k = len(q)
            xi = kept.pop()
            rest = [a for a in range(n) if a not in q]
            dp = torch.tensordot(g, xi, dims=(rest, rest)).reshape(-1)
            # tensordot lists the kept axes in ascending order, as q is
            row = torch.zeros(256, dtype=torch.float64, device='cuda')
            row[:dp.numel()] = dp
            rows.append(row)
            g = _apply(g, p.permute(list(range(k, 2 * k)) +
                                    list(range(k))).contiguous(), q)
        grads += rows[::-1]
    return {'prob': torch.cat(probs), 'loss': torch.stack(losses),
            'grads': torch.stack(grads)}


def exact(case, seed):
    kind = case['kind']
    if kind == 'grad':
        return _exact_grad(case, seed)
    if kind == 'batch':
        with torch.no_grad():
            return _exact_batch(case, seed)
    n, d = case['n'], 3 if kind.startswith('qutrits') else 2
    x = _state(n, d, seed, _dtype(case)).double()
    if kind == 'readout':
        return _exact_readout(case, x)
    gates = [(torch.from_numpy(p).cuda(), qs) for p, qs in _gates(case, seed)]
    if kind == 'diff':
        x.requires_grad_(True)
        gates = [(p.requires_grad_(True), qs) for p, qs in gates]
    y = functools.reduce(lambda s, g: _apply(s, *g), gates, x)
    if kind == 'diff':
        t = _histogram(np.random.default_rng([seed, 9]), 2 ** n).cuda()
        prob = y.reshape(-1)[_diag_index(n)]
        loss = _loss(prob, t)
        grads = torch.autograd.grad(loss, [x] + [p for p, _ in gates])
        return {'loss': loss.detach(), 'prob': prob.detach(), 'grads': grads}
    if kind == 'fused':
        red, keep = y, _choice(case, 4)
        for q in reversed(range(n)):
            if q not in keep:
                red = red.select(q, 0) + red.select(q, 1)
        return {'state': y, 'reduced': red}
    if kind == 'units':
        return {'state': y, 'diagonal': y.reshape(-1)[_diag_index(n)]}
    if kind == 'qutrits':
        # per qutrit, the first three basis elements are the projectors
        diag = y
        for a in range(n):
            diag = diag.narrow(a, 0, 3)
        q = _choice(case, 1)[0]
        probs = diag.sum(dim=[a for a in range(n) if a != q])
        k = int(torch.argmax(probs))
        return {'probs': probs, 'weight': float(probs[k]),
                'state': y.narrow(q, k, 1) / probs[k]}
    return y

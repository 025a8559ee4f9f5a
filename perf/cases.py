"""Work that users of this package have it do, as cases that can be timed.

listed()             the named cases
draw(rng)            one more case of the same ranges
prepare(case, seed)  what a program holds before the call
run(state)           one pass through the public entry points, and its outputs
work(case)           bytes and operations one pass cannot do without
exact(case, seed)    run()'s outputs in 64-bit arithmetic (numpy / torch), where that is quick

The kinds of case:

run       ``hpc.bond_microcanonical_statistics`` for one numpy seed
task      one task of the reference's job: one run's rows, their canonical
          statistics at every p, and the merge into the running averages
classic   ``percolate.statistics``: canonical averages of a few runs of a graph
ensemble  ``Ensemble.run`` with the finalised canonical averages and the
          microcanonical averages of every n read back
mix       ``MixEnsemble.run``: runs of unequal lattices in one launch
mlp       one training step of the surrogate network
"""
import math

import numpy as np
import torch

from pypercolate_gb300 import hpc, percolate
from pypercolate_gb300.ensemble import Ensemble
from pypercolate_gb300.mix import MixEnsemble
from pypercolate_gb300.surrogate import MLP, WIDTHS


def listed():
    return [
        # the smallest call: one run of the 16 x 16 grid by numpy seed (the plain method's lattice)
        {'name': 'run grid 16', 'kind': 'run', 'length': 16},
        # the same call on a large lattice of odd size
        {'name': 'run grid 181', 'kind': 'run', 'length': 181},
        # one task of a job over seeds: run, canonical statistics at 101 p, merge, finalise
        {'name': 'task grid 48', 'kind': 'task', 'length': 48, 'points': 101},
        # the classic interface with its default of 40 runs
        {'name': 'classic grid 40', 'kind': 'classic', 'length': 40, 'runs': 40, 'points': 101},
        # a quick look at a small lattice: a thousand runs
        {'name': 'ensemble grid 32', 'kind': 'ensemble', 'lattice': 'grid', 'model': 'bond', 'wrap': 'either',
         'length': 32, 'runs': 1000, 'points': 201, 'precision': 'fp32'},
        # one lattice of a finite-size-scaling series, its size no power of two
        {'name': 'ensemble grid 97', 'kind': 'ensemble', 'lattice': 'grid', 'model': 'bond', 'wrap': 'either',
         'length': 97, 'runs': 4000, 'points': 501, 'precision': 'fp32'},
        # the benchmark's lattice and p-grid with tens of thousands of runs
        {'name': 'ensemble grid 256', 'kind': 'ensemble', 'lattice': 'grid', 'model': 'bond', 'wrap': 'either',
         'length': 256, 'runs': 40000, 'points': 1001, 'precision': 'fp32'},
        # a large lattice with few runs, convolved on the tensor cores
        {'name': 'ensemble grid 512 tf32x3', 'kind': 'ensemble', 'lattice': 'grid', 'model': 'bond', 'wrap': 'either',
         'length': 512, 'runs': 200, 'points': 501, 'precision': 'tf32x3'},
        # chains, convolved in FP64
        {'name': 'ensemble chain 6000 fp64', 'kind': 'ensemble', 'lattice': 'chain', 'model': 'bond',
         'wrap': 'either', 'length': 6000, 'runs': 3000, 'points': 201, 'precision': 'fp64'},
        # wrapping probabilities on the torus
        {'name': 'ensemble torus 64', 'kind': 'ensemble', 'lattice': 'torus', 'model': 'bond', 'wrap': 'both',
         'length': 64, 'runs': 5000, 'points': 301, 'precision': 'fp32'},
        # the batched uneven workload, a tenth of its benchmark size
        {'name': 'mix 100000', 'kind': 'mix', 'runs': 100000, 'grid_max': 512, 'chain_max': 65536,
         'checkpoints': 256, 'fused': False},
        # one training step of the surrogate at its batch size
        {'name': 'mlp step 4096', 'kind': 'mlp', 'batch': 4096, 'weighted': True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['run', 'task', 'classic', 'ensemble', 'ensemble', 'ensemble', 'ensemble', 'mix', 'mlp'])
    if kind == 'run':
        return {'kind': kind, 'length': _log_int(rng, 8, 181)}
    if kind == 'task':
        return {'kind': kind, 'length': _log_int(rng, 8, 64), 'points': _log_int(rng, 20, 201)}
    if kind == 'classic':
        return {'kind': kind, 'length': _log_int(rng, 8, 64), 'runs': _log_int(rng, 10, 80),
                'points': _log_int(rng, 20, 201)}
    if kind == 'mix':
        return {'kind': kind, 'runs': _log_int(rng, 2000, 100000), 'grid_max': _log_int(rng, 32, 512),
                'chain_max': _log_int(rng, 2048, 65536), 'checkpoints': rng.choice([64, 101, 256]),
                'fused': rng.random() < 0.5}
    if kind == 'mlp':
        return {'kind': kind, 'batch': _log_int(rng, 256, 8192), 'weighted': rng.random() < 0.5}
    lattice, model, wrap = rng.choice([('grid', 'bond', 'either')] * 3 + [
        ('chain', 'bond', 'either'), ('torus', 'bond', rng.choice(['either', 'x', 'y', 'both'])),
        ('grid', 'site', 'either'), ('torus', 'site', 'either'), ('chain', 'site', 'either')])
    precision = rng.choice(['fp32', 'fp32', 'tf32x3', 'fp64'])
    length = _log_int(rng, 200, 20000) if lattice == 'chain' else _log_int(rng, 8, 320)
    sites = length if lattice == 'chain' else length * length
    # no more than the largest listed case: steps of all runs, and their records
    runs = _log_int(rng, 100, max(101, min(40000, int(1.2e9 / sites))))
    return {'kind': kind, 'lattice': lattice, 'model': model, 'wrap': wrap, 'length': length, 'runs': runs,
            'points': _log_int(rng, 20, 600), 'precision': precision}


# ------------------------------------------------------------------ sizes
def _size(case):
    """(nodes, steps of one run)."""
    length = case['length']
    lattice, site = case.get('lattice', 'grid'), case.get('model') == 'site'
    if lattice == 'chain':
        nodes, bonds = length, length - 1
    else:
        nodes = length * length
        bonds = 2 * nodes if lattice == 'torus' else 2 * length * (length - 1)
    return nodes, nodes if site else bonds


def _ps(points):
    return np.linspace(0.0, 1.0, points)


def _band_terms(steps, points):
    """Terms of the canonical sums of one run and statistic: the rows within
    +-7.7 standard deviations of n = p M, which hold all but 1e-13 of the
    binomial weight."""
    ps = _ps(points)
    return float(np.minimum(15.4 * np.sqrt(steps * ps * (1.0 - ps)) + 1.0, steps + 1.0).sum())


# operations of one step of a run: draw its bond, two finds, the union and
# the update of seven statistics
STEP_OPS = 30


def work(case):
    kind = case['kind']
    if kind == 'mlp':
        batch, weights = case['batch'], sum(a * b for a, b in zip(WIDTHS[:-1], WIDTHS[1:]))
        params = weights + sum(WIDTHS[1:])
        return {'bytes': 4.0 * (batch * (WIDTHS[0] + 3 * WIDTHS[-1]) + 8 * params),
                'flops': 6.0 * batch * weights - 2.0 * batch * WIDTHS[0] * WIDTHS[1]}
    if kind == 'mix':
        # log-uniform lengths: the mean of l over [a, b] is (b - a) / ln(b / a)
        g, c, f = case['grid_max'], case['chain_max'], case['checkpoints']
        steps = 0.5 * (g * g - 64.0) / math.log(g / 8.0) + 0.5 * (c - 1024.0) / math.log(c / 1024.0)
        classes = (g - 7) + (c - 1023)
        return {'bytes': classes * f * 148.0, 'flops': STEP_OPS * case['runs'] * steps}
    nodes, steps = _size(case)
    rows = steps + 1
    if kind == 'run':
        return {'bytes': 53.0 * rows, 'flops': float(STEP_OPS * steps)}
    points = case['points']
    if kind == 'task':
        return {'bytes': 53.0 * rows + 8.0 * points * rows + 4 * 116.0 * points,
                'flops': STEP_OPS * steps + 14.0 * points * rows}
    runs = case['runs']
    if kind == 'classic':
        return {'bytes': 8.0 * 21 * points,
                'flops': STEP_OPS * steps * runs + 2.0 * 21 * _band_terms(steps, points)}
    return {'bytes': 8.0 * 21 * rows + 8.0 * 31 * points,
            'flops': runs * (STEP_OPS * steps + 14.0 * _band_terms(steps, points))}


# ------------------------------------------------------------------ prepare
def _mlp_data(case, seed):
    """Standardised inputs of the surrogate's network with smooth targets."""
    gen = torch.Generator(device='cuda')
    gen.manual_seed(seed)
    b = case['batch']
    x = torch.randn(b, WIDTHS[0], device='cuda', generator=gen)
    x[:, 2] = torch.where(x[:, 2] > 0, 1.0, -1.0)
    x[:, 3] = -x[:, 2]
    t = torch.stack([torch.tanh(x[:, 4] + 0.3 * x[:, 2]), 0.7 * x[:, 0] - 0.2 * x[:, 1],
                     torch.cos(x[:, 4]) + 0.1 * x[:, 0]], dim=1).contiguous()
    w = None
    if case['weighted']:
        w = torch.exp(0.8 * torch.randn(b, WIDTHS[-1], device='cuda', generator=gen))
    return x.contiguous(), t, w


def prepare(case, seed):
    kind = case['kind']
    state = {'kind': kind, 'seed': int(seed)}
    if kind == 'run' or kind == 'task':
        state['graph'] = percolate.percolation_graph(percolate.spanning_2d_grid(case['length']))
    if kind == 'task':
        points = case['points']
        nodes, steps = _size(case)
        state['ps'] = _ps(points)
        # the job computes its convolution factors once
        state['factors'] = percolate.binomial_pmfs(steps, state['ps'])
        # averages of the runs that came before
        rng = np.random.default_rng(seed)
        stats = np.zeros(points, dtype=hpc.canonical_statistics_dtype(True))
        stats['percolation_probability'] = rng.random(points)
        stats['max_cluster_size'] = nodes * rng.random(points)
        stats['moments'] = (nodes * rng.random((points, 1))) ** np.array([[0.5, 1.0, 1.5, 2.0, 2.5]])
        state['averages'] = hpc.bond_initialize_canonical_averages(stats)
    elif kind == 'classic':
        state['graph'] = percolate.spanning_2d_grid(case['length'])
        state['ps'] = _ps(case['points'])
        state['runs'] = case['runs']
    elif kind == 'ensemble':
        state['ensemble'] = Ensemble(case['lattice'], case['length'], _ps(case['points']),
                                     precision=case['precision'], model=case['model'], wrap=case['wrap'])
        state['runs'], state['run0'] = case['runs'], 0
    elif kind == 'mix':
        state['mix'] = MixEnsemble(case['runs'], grid=(8, case['grid_max']), chain=(1024, case['chain_max']),
                                   checkpoints=case['checkpoints'], fused=case['fused'])
    elif kind == 'mlp':
        state['mlp'] = MLP(seed=seed)
        state['data'] = _mlp_data(case, seed)
    return state


# ---------------------------------------------------------------------- run
def _fields(rows):
    return {name: rows[name] for name in rows.dtype.names}


def run(state):
    kind = state['kind']
    if kind == 'run':
        return _fields(hpc.bond_microcanonical_statistics(seed=state['seed'], **state['graph']))
    if kind == 'task':
        rows = hpc.bond_microcanonical_statistics(seed=state['seed'], **state['graph'])
        stats = hpc.bond_canonical_statistics(rows, state['factors'])
        averages = hpc.bond_reduce(state['averages'], hpc.bond_initialize_canonical_averages(stats))
        final = hpc.finalize_canonical_averages(state['graph']['num_nodes'], state['ps'], averages, 0.05)
        return {'rows': _fields(rows), 'statistics': _fields(stats), 'averages': _fields(averages),
                'final': _fields(final)}
    if kind == 'classic':
        np.random.seed(state['seed'])
        return percolate.statistics(state['graph'], state['ps'], runs=state['runs'])
    if kind == 'ensemble':
        ens = state['ensemble']
        ens.run(state['runs'], key=state['seed'], run0=state['run0'])
        state['run0'] += state['runs']
        return {'canonical': _fields(ens.finalized()), 'microcanonical': ens.microcanonical_averages()}
    if kind == 'mix':
        mix = state['mix'].run(state['seed'])
        return {'count': mix.count, 'span': mix.span, 'sum_lo': mix.sum_lo, 'sum_hi': mix.sum_hi, 'm2': mix.m2,
                'errors': mix.errors}
    x, t, w = state['data']
    net = state['mlp']
    loss = net.loss_and_grads(x, t, w)
    net.adam()
    return {'loss': loss, 'grads': net.grads, 'params': net.params}


# -------------------------------------------------------------------- exact
def _lowbias32(x):
    x ^= x >> np.uint32(16)
    x *= np.uint32(0x7feb352d)
    x ^= x >> np.uint32(15)
    x *= np.uint32(0x846ca68b)
    x ^= x >> np.uint32(16)
    return x


def _philox(c, k0, k1):
    c = [np.asarray(v, dtype=np.uint64) for v in c]
    mask = np.uint64(0xffffffff)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return [v.astype(np.uint32) for v in c]


def _permutations(steps, runs, key):
    """The keyed permutations of the run ids 0 .. runs - 1, shape (steps, runs)."""
    ids = np.arange(runs, dtype=np.uint64)
    keys = []
    for half in (0, 1):
        c = [ids, np.zeros_like(ids), np.full_like(ids, half), np.full_like(ids, 0x5045524D)]
        keys += _philox(c, key & 0xffffffff, key >> 32)
    bits = int(steps - 1).bit_length() if steps > 1 else 0
    hl, hr = bits // 2, bits - bits // 2

    def part(v, width, k):
        return _lowbias32(v ^ k) >> np.uint32(32 - width) if width else np.zeros_like(v)

    def encrypt(x, cols):
        left, right = x >> np.uint32(hr), x & np.uint32((1 << hr) - 1)
        for i in range(0, 8, 2):
            left = left ^ part(right, hl, keys[i][cols])
            right = right ^ part(left, hr, keys[i + 1][cols])
        return (left << np.uint32(hr)) | right

    rows, cols = np.meshgrid(np.arange(steps, dtype=np.uint32), np.arange(runs), indexing='ij')
    x = encrypt(rows, cols)
    walk = x >= steps
    while walk.any():
        x[walk] = encrypt(x[walk], cols[walk])
        walk = x >= steps
    return x


def _grid_edges(length):
    """Bonds of the grid, node-major: to the next row, then to the next column."""
    u, v = [], []
    for i in range(length):
        for j in range(length):
            k = i * length + j
            if i < length - 1:
                u.append(k)
                v.append(k + length)
            if j < length - 1:
                u.append(k)
                v.append(k + 1)
    return np.array(u, dtype=np.int64), np.array(v, dtype=np.int64)


def _sample(case, perms):
    """Statistics of bond percolation after every step, one array
    (steps + 1, runs) each: spanning, max, moments 0 .. 4 without the largest."""
    nodes, steps = _size(case)
    length = case['length']
    side = np.zeros(nodes, dtype=np.int64)
    if case.get('lattice') == 'chain':
        u, v = np.arange(steps), np.arange(1, steps + 1)
        side[0], side[-1] = 1, side[-1] | 2
    else:
        u, v = _grid_edges(length)
        side[:length] |= 1
        side[nodes - length:] |= 2
    runs = perms.shape[1]
    at = np.arange(runs)
    parent = np.tile(np.arange(nodes), (runs, 1))
    size = np.ones((runs, nodes), dtype=np.int64)
    sides = np.tile(side, (runs, 1))
    out = np.zeros((steps + 1, 7, runs))
    totals = np.full((5, runs), float(nodes))  # sums of size^k over all clusters
    largest = np.ones(runs)
    span = np.zeros(runs)
    powers = np.arange(5)[:, None]

    def find(x):
        while True:
            up = parent[at, x]
            if (up == x).all():
                return x
            parent[at, x] = parent[at, up]
            x = up

    for n in range(steps + 1):
        if n:
            e = perms[n - 1]
            a, b = find(u[e]), find(v[e])
            sa, sb = size[at, a], size[at, b]
            swap = sa < sb
            a, b = np.where(swap, b, a), np.where(swap, a, b)
            new = a != b
            both = np.where(new, sa + sb, sa)
            parent[at[new], b[new]] = a[new]
            size[at, a] = both
            sides[at, a] |= sides[at, b]
            span = np.maximum(span, (new & (sides[at, a] == 3)).astype(float))
            fa, fb = sa.astype(float), sb.astype(float)
            totals += np.where(new, (fa + fb) ** powers - fa ** powers - fb ** powers, 0.0)
            largest = np.maximum(largest, both)
        out[n, 0], out[n, 1] = span, largest
        out[n, 2:] = totals - largest ** powers
    return out


def _weights(steps, ps):
    n = np.arange(steps + 1, dtype=np.float64)
    log_factorial = np.concatenate([[0.0], np.cumsum(np.log(np.arange(1, steps + 1, dtype=np.float64)))])
    shape = -log_factorial - log_factorial[::-1]
    w = np.zeros((len(ps), steps + 1))
    for i, p in enumerate(ps):
        if p <= 0.0 or p >= 1.0:
            w[i, 0 if p <= 0.0 else steps] = 1.0
        else:
            x = shape + n * math.log(p) + (steps - n) * math.log1p(-p)
            x = np.exp(x - x.max())
            w[i] = x / x.sum()
    return w


def _exact_ensemble(case, seed):
    nodes, steps = _size(case)
    runs, ps = case['runs'], _ps(case['points'])
    if case['model'] != 'bond' or case['lattice'] == 'torus' or runs < 2 or steps > 2500 or runs * steps > 4e6:
        return None
    micro = _sample(case, _permutations(steps, runs, int(seed)))
    stats = np.tensordot(_weights(steps, ps), micro, axes=(1, 0))  # (p, statistic, run)
    mean, std = stats.mean(axis=2), stats.std(axis=2, ddof=1)
    mean[:, 1:] /= nodes
    std[:, 1:] /= nodes
    means = micro.mean(axis=2) / nodes
    return {'canonical': {'number_of_runs': None, 'p': ps, 'alpha': None, 'percolation_probability_mean': mean[:, 0],
                          'percolation_probability_std': std[:, 0], 'percolation_probability_ci': None,
                          'percolation_strength_mean': mean[:, 1], 'percolation_strength_std': std[:, 1],
                          'percolation_strength_ci': None, 'moments_mean': mean[:, 2:], 'moments_std': std[:, 2:],
                          'moments_ci': None},
            'microcanonical': {'N': None, 'M': None,
                               'spanning_cluster': (micro[:, 0].sum(axis=1) + 1.0) / (runs + 2.0),
                               'spanning_cluster_ci': None, 'max_cluster_size': means[:, 1],
                               'max_cluster_size_ci': None, 'moments': means[:, 2:].T.copy(), 'moments_ci': None}}


def _exact_classic(case, seed):
    nodes, steps = _size(case)
    runs, ps = case['runs'], _ps(case['points'])
    if steps > 5000:
        return None
    rng = np.random.RandomState(int(seed))
    micro = _sample(case, np.stack([rng.permutation(steps) for _ in range(runs)], axis=1))
    w = _weights(steps, ps)
    means = w @ (micro.mean(axis=2) / nodes)
    return {'ps': ps, 'N': None, 'M': None, 'max_cluster_size': means[:, 1], 'max_cluster_size_ci': None,
            'moments': means[:, 2:].T.copy(), 'moments_ci': None,
            'spanning_cluster': w @ ((micro[:, 0].sum(axis=1) + 1.0) / (runs + 2.0)), 'spanning_cluster_ci': None}


def _exact_task(case, seed):
    nodes, steps = _size(case)
    ps = _ps(case['points'])
    perm = np.random.RandomState(int(seed)).permutation(steps)[:, None]
    stats = _weights(steps, ps) @ _sample(case, perm)[:, :, 0]
    rng = np.random.default_rng(int(seed))
    before = np.empty((case['points'], 7))
    before[:, 0] = rng.random(case['points'])
    before[:, 1] = nodes * rng.random(case['points'])
    before[:, 2:] = (nodes * rng.random((case['points'], 1))) ** np.array([[0.5, 1.0, 1.5, 2.0, 2.5]])
    mean = 0.5 * (stats + before)
    m2 = 0.5 * (stats - before) ** 2
    norm = np.array([1.0] + [float(nodes)] * 6)
    fmean, fstd = mean / norm, np.sqrt(m2) / norm
    return {'rows': {'n': None, 'edge': None, 'has_spanning_cluster': None, 'max_cluster_size': None, 'moments': None},
            'statistics': {'percolation_probability': stats[:, 0], 'max_cluster_size': stats[:, 1],
                           'moments': stats[:, 2:]},
            'averages': {'number_of_runs': None, 'percolation_probability_mean': mean[:, 0],
                         'percolation_probability_m2': m2[:, 0], 'max_cluster_size_mean': mean[:, 1],
                         'max_cluster_size_m2': m2[:, 1], 'moments_mean': mean[:, 2:], 'moments_m2': m2[:, 2:]},
            'final': {'number_of_runs': None, 'p': ps, 'alpha': None, 'percolation_probability_mean': fmean[:, 0],
                      'percolation_probability_std': fstd[:, 0], 'percolation_probability_ci': None,
                      'percolation_strength_mean': fmean[:, 1], 'percolation_strength_std': fstd[:, 1],
                      'percolation_strength_ci': None, 'moments_mean': fmean[:, 2:], 'moments_std': fstd[:, 2:],
                      'moments_ci': None}}


def _exact_mlp(case, seed):
    x, t, w = _mlp_data(case, seed)
    # the initial parameters as MLP draws them: uniform weights, zero biases
    rng = np.random.default_rng(int(seed))
    params = []
    for a, b in zip(WIDTHS[:-1], WIDTHS[1:]):
        bound = np.sqrt(6.0 / a) / np.sqrt(2.0)
        params.append(rng.uniform(-bound, bound, a * b).astype(np.float32).astype(np.float64))
        params.append(np.zeros(b))
    leaves = [torch.tensor(p, dtype=torch.float64, device='cuda', requires_grad=True) for p in params]
    h = x.double()
    layers = len(WIDTHS) - 1
    for i in range(layers):
        h = h @ leaves[2 * i].view(WIDTHS[i], WIDTHS[i + 1]) + leaves[2 * i + 1]
        if i < layers - 1:
            h = torch.nn.functional.gelu(h)
    err = (h - t.double()) ** 2
    loss = (err if w is None else err * w.double()).sum() / case['batch']
    loss.backward()
    g = torch.cat([p.grad for p in leaves])
    p = torch.cat([p.detach() for p in leaves])
    return {'loss': loss.detach(), 'grads': g, 'params': p - 1e-3 * g / (g.abs() + 1e-8)}


def exact(case, seed):
    kind = case['kind']
    if kind == 'ensemble':
        return _exact_ensemble(case, seed)
    if kind == 'classic':
        return _exact_classic(case, seed)
    if kind == 'task':
        return _exact_task(case, seed)
    if kind == 'mlp':
        return _exact_mlp(case, seed)
    return None

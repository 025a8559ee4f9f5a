"""Union-find with a thread block per run: exact integers at the sizes where
its batches, node formats and claims change, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from pypercolate_gb300 import _native as nat
    nat.lib_handle()
    return nat


def _check(host, r, ref):
    assert np.array_equal(host['max_span'][:, r] & 0x7fffffff, ref['max'])
    assert np.array_equal((host['max_span'][:, r] >> 31).astype(bool), ref['span'])
    assert np.array_equal(host['m0'][:, r], ref['moments_u64'][:, 0])
    assert np.array_equal(host['m2'][:, r], ref['moments_u64'][:, 2])
    assert np.array_equal(host['m3'][:, r], ref['moments_u64'][:, 3])
    assert np.array_equal(host['m4_lo'][:, r], ref['moments_u64'][:, 4])
    assert np.array_equal(host['edge'][1:, r], ref['edge'][1:])


# 1 to 16 warps per run (few and many runs of small and large lattices), the
# last grid (256) and chain (65,536) in shared memory, the first beyond
@pytest.mark.parametrize('kind,L,runs', [
    (0, 2, 3), (0, 3, 700), (0, 9, 5000), (0, 23, 40), (0, 40, 1500), (0, 64, 20), (0, 100, 3), (0, 256, 2),
    (0, 257, 2), (1, 2, 9), (1, 33, 3000), (1, 65536, 1), (1, 65537, 1)])
def test_records_match_oracle(gpu, oracle, kind, L, runs):
    from pypercolate_gb300 import hpc
    spec = hpc.GraphSpec((gpu.GRAPH_GRID2D, gpu.GRAPH_CHAIN1D)[kind], L)
    rec = hpc._run_microcanonical(spec, True, rng='philox', key=17, run0=5, n_runs=runs)
    host = rec.host()
    for r in sorted({0, runs // 2, runs - 1}):
        _check(host, r, oracle.lattice_run((oracle.GRID_2D, oracle.CHAIN_1D)[kind], L,
                                           oracle.philox_permutation(17, 5 + r, spec.M)))


@pytest.mark.parametrize('order', ['forward', 'backward', 'inside out'])
@pytest.mark.parametrize('L', [5, 300, 70000])
def test_chain_in_order(gpu, oracle, order, L):
    """Every bond of a batch depends on the one before it."""
    from pypercolate_gb300 import hpc
    spec = hpc.GraphSpec(gpu.GRAPH_CHAIN1D, L)
    perm = np.arange(spec.M, dtype=np.uint32)
    if order == 'backward':
        perm = perm[::-1].copy()
    elif order == 'inside out':
        perm = perm[np.argsort(np.abs(perm.astype(np.int64) - spec.M // 2), kind='stable')]
    rec = hpc._run_microcanonical(spec, True, perms=perm[None])
    _check(rec.host(), 0, oracle.lattice_run(oracle.CHAIN_1D, L, perm))


@pytest.mark.parametrize('N,M', [(7, 40), (1000, 3000), (70000, 9000)])
def test_random_edge_lists(gpu, oracle, N, M):
    """Self-loops, repeated edges and nodes on one side, the other or neither."""
    from pypercolate_gb300 import hpc
    rng = np.random.default_rng(N)
    eu, ev = (rng.integers(0, N, M).astype(np.uint32) for _ in range(2))
    hub = rng.random(M) < 0.3
    eu[hub] = N // 2
    side = rng.choice([0, 0, 0, 1, 2], N).astype(np.uint8)
    perms = np.stack([rng.permutation(M) for _ in range(3)]).astype(np.uint32)
    spec = hpc.GraphSpec(gpu.GRAPH_EDGES, 0, N, M, eu, ev, side)
    host = hpc._run_microcanonical(spec, True, perms=perms).host()
    for r in range(3):
        _check(host, r, oracle.sample_states(N, M, eu, ev, side, True, perms[r]))


@pytest.mark.parametrize('kind,L,window', [('grid', 30, 70), ('grid', 30, 33), ('chain', 900, 256), ('grid', 258, 40000)])
def test_windows_leave_the_sums_alone(gpu, kind, L, window):
    """Node words and totals carried from window to window; rows that are no
    multiple of 32 or of a batch."""
    from pypercolate_gb300.ensemble import Ensemble
    ps = np.array([0.3, 0.5, 0.9])
    got = []
    for w in (0, window):
        e = Ensemble(kind, L, ps, precision='fp64', window=w)
        e.run(50, key=3)
        assert e.errors() == 0
        got.append((e.micro_sums(), e.mean.cpu().numpy()))
    (a, ma), (b, mb) = got
    assert np.array_equal(a['span_count'], b['span_count'])
    assert (a['sums'] == b['sums']).all()
    np.testing.assert_array_equal(a['m2'], b['m2'])
    np.testing.assert_allclose(ma, mb, rtol=1e-12)  # FP64 sums of < 2^17 terms in another order


# 128: the last torus in shared memory; wrapping criteria, and one and two
# nodes to a side, where bonds are loops and doubled
@pytest.mark.parametrize('wrap', ['either', 'x', 'y', 'both'])
@pytest.mark.parametrize('L,runs', [(1, 2), (2, 40), (3, 2000), (20, 60), (33, 700), (128, 2), (129, 2)])
def test_torus_matches_census(gpu, oracle, L, runs, wrap):
    from pypercolate_gb300 import lattice
    host = lattice.sample_records('torus', L, wrap=wrap, n_runs=runs, key=23, run0=3)
    M = 2 * L * L
    for r in sorted({0, runs - 1} if L < 100 else {runs - 1}):
        perm = oracle.philox_permutation(23, 3 + r, M)
        assert np.array_equal(host['edge'][1:, r], perm)
        if L <= 33:  # the census is a search of the lattice per step
            ref = oracle.lattice_census('torus', L, perm, wrap=wrap)
            for plane in ('max_span', 'm0', 'm2', 'm3', 'm4_lo'):
                assert np.array_equal(host[plane][:, r], ref[plane]), plane
        else:
            eu, ev = _torus_edges(L)
            ref = oracle.sample_states(L * L, M, eu, ev, np.zeros(L * L, np.uint8), False, perm)
            assert np.array_equal(host['max_span'][:, r] & 0x7fffffff, ref['max'])
            assert np.array_equal(host['m4_lo'][:, r], ref['moments_u64'][:, 4])
            assert np.array_equal((host['max_span'][:, r] >> 31).astype(bool), _wraps(L, perm, wrap))


def _torus_edges(L):
    n = np.arange(L * L)
    row, col = n // L, n % L
    return (np.concatenate([n, n]).astype(np.uint32),
            np.concatenate([row * L + (col + 1) % L, (row + 1) % L * L + col]).astype(np.uint32))


def _wraps(L, perm, wrap):
    """Wrapping flags by a union-find with positions, one bond at a time."""
    N = L * L
    eu, ev = (a.astype(int).tolist() for a in _torus_edges(L))
    parent, off, size = list(range(N)), [(0, 0)] * N, [1] * N
    wx = wy = False
    out = [False]
    for e in perm.tolist():
        u, v, pos = eu[e], ev[e], []
        for x in (u, v):
            px = py = 0
            while parent[x] != x:
                px, py, x = px + off[x][0], py + off[x][1], parent[x]
            pos.append((x, px, py))
        (a, ax, ay), (b, bx, by) = pos
        dx, dy = ax + (e < N) - bx, ay + (e >= N) - by
        if a == b:
            wx, wy = wx or dx != 0, wy or dy != 0
        elif size[a] >= size[b]:
            parent[b], off[b], size[a] = a, (dx, dy), size[a] + size[b]
        else:
            parent[a], off[a], size[b] = b, (-dx, -dy), size[a] + size[b]
        out.append({'either': wx or wy, 'x': wx, 'y': wy, 'both': wx and wy}[wrap])
    return np.array(out)


def test_torus_windows(gpu):
    from pypercolate_gb300.ensemble import Ensemble
    for L, window in ((24, 100), (130, 20000)):
        got = []
        for w in (0, window):
            e = Ensemble('torus', L, [0.4, 0.5], precision='fp64', wrap='both', window=w)
            e.run(40, key=3)
            assert e.errors() == 0
            got.append(e.micro_sums())
        assert np.array_equal(got[0]['span_count'], got[1]['span_count'])
        assert (got[0]['sums'] == got[1]['sums']).all()


def _site_run(kind, L, perm, wrap):
    """Site percolation, one site at a time: max, flag, m0 and sums of powers."""
    N = L if kind == 'chain' else L * L
    height, width = (1, L) if kind == 'chain' else (L, L)
    parent, off, size, sides = list(range(N)), [(0, 0)] * N, [0] * N, [0] * N
    wx = wy = span = False
    total, clusters, most = [0, 0, 0], 0, 0
    out = [(0, False, 0, 0, 0, 0)]
    for s in perm:
        if s < N and size[s] == 0 and parent[s] == s:
            row, col = s // width, s % width
            size[s] = 1
            if kind != 'torus':
                at, end = (row, height) if kind == 'grid' else (col, width)
                sides[s] = (1 if at == 0 else 0) | (2 if at == end - 1 else 0)
            total = [t + 1 for t in total]
            clusters += 1
            most = max(most, 1)
            span = span or sides[s] == 3
            for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1)):
                r, c = row + dy, col + dx
                if kind == 'torus':
                    r, c = r % L, c % L
                elif not (0 <= r < height and 0 <= c < width):
                    continue
                v = r * width + c
                if size[v] == 0 and parent[v] == v:
                    continue
                pos = []
                for x in (s, v):
                    px = py = 0
                    while parent[x] != x:
                        px, py, x = px + off[x][0], py + off[x][1], parent[x]
                    pos.append((x, px, py))
                (a, ax, ay), (b, bx, by) = pos
                ox, oy = ax + dx - bx, ay + dy - by
                if a == b:
                    wx, wy = wx or ox != 0, wy or oy != 0
                    continue
                if size[a] < size[b]:
                    a, b, ox, oy = b, a, -ox, -oy
                total = [t + (size[a] + size[b]) ** k - size[a] ** k - size[b] ** k
                         for t, k in zip(total, (2, 3, 4))]
                parent[b], off[b] = a, (ox, oy)
                size[a] += size[b]
                sides[a] |= sides[b]
                clusters -= 1
                most = max(most, size[a])
                span = span or sides[a] == 3
        flag = {'either': wx or wy, 'x': wx, 'y': wy, 'both': wx and wy}[wrap] if kind == 'torus' else span
        out.append((most, flag, max(clusters - 1, 0)) + tuple(t - most ** k for t, k in zip(total, (2, 3, 4))))
    return out


@pytest.mark.parametrize('kind,L,runs', [
    ('grid', 2, 3), ('grid', 3, 700), ('grid', 9, 5000), ('grid', 23, 40), ('grid', 100, 3), ('grid', 256, 1),
    ('grid', 257, 1), ('chain', 3, 900), ('chain', 65536, 1), ('chain', 65537, 1), ('torus', 3, 2000),
    ('torus', 24, 60), ('torus', 128, 2), ('torus', 129, 1)])
@pytest.mark.parametrize('order', ['keyed', 'given'])
def test_site_records(gpu, oracle, kind, L, runs, order):
    """Occupied sites claim themselves and their neighbours' clusters; a
    caller's order may name sites twice or none at all."""
    from pypercolate_gb300 import lattice
    N = L if kind == 'chain' else L * L
    wrap = 'both' if kind == 'torus' else 'either'
    runs = runs if order == 'keyed' else 2
    if order == 'keyed':
        host = lattice.sample_records(kind, L, 'site', wrap, n_runs=runs, key=41, run0=7)
        perm = oracle.philox_permutation(41, 7 + runs - 1, N)
    else:
        rng = np.random.default_rng(L)
        perms = np.stack([rng.permutation(N) for _ in range(runs)]).astype(np.uint32)
        perms[:, N // 3:2 * N // 3] = rng.integers(0, N + 2, (runs, 2 * N // 3 - N // 3))
        host = lattice.sample_records(kind, L, 'site', wrap, perms=perms)
        perm = perms[-1]
    want = _site_run(kind, L, perm.tolist(), wrap)
    r = runs - 1
    assert np.array_equal(host['edge'][1:, r], perm)
    assert np.array_equal(host['max_span'][:, r] & 0x7fffffff, [w[0] for w in want])
    assert np.array_equal((host['max_span'][:, r] >> 31).astype(bool), [w[1] for w in want])
    assert np.array_equal(host['m0'][:, r], [w[2] for w in want])
    assert host['m2'][:, r].tolist() == [w[3] for w in want]
    assert host['m3'][:, r].tolist() == [w[4] for w in want]
    m4 = [int(a) | int(b) << 64 for a, b in zip(host['m4_lo'][:, r], host['m4_hi'][:, r])]
    assert m4 == [w[5] for w in want]


@pytest.mark.parametrize('kind,L,window', [('grid', 30, 70), ('chain', 900, 256), ('grid', 258, 40000), ('torus', 24, 100),
                                           ('torus', 130, 9000), ('chain', 1, 1), ('grid', 1, 1), ('torus', 1, 1),
                                           ('chain', 2, 1)])
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
def test_site_windows(gpu, kind, L, window, precision):
    from pypercolate_gb300.ensemble import Ensemble
    ps = np.array([0.3, 0.55, 0.6, 0.9])
    got = []
    for w in (0, window):
        e = Ensemble(kind, L, ps, precision=precision, model='site', window=w)
        e.run(40, key=3)
        assert e.errors() == 0
        got.append((e.micro_sums(), e.mean.cpu().numpy()))
    (a, ma), (b, mb) = got
    assert np.array_equal(a['span_count'], b['span_count'])
    assert (a['sums'] == b['sums']).all()
    # FP64: sums of < 2^17 terms in another order; FP32: partial sums of 128 rows
    # cut elsewhere, each within 128 * 2^-24 of exact
    np.testing.assert_allclose(ma, mb, rtol=1e-12 if precision == 'fp64' else 2e-5)


@pytest.mark.parametrize('precision', ['fp32', 'tf32x3'])
@pytest.mark.parametrize('kind,L,model', [('grid', 24, 'bond'), ('grid', 90, 'site'), ('grid', 345, 'bond'),
                                          ('chain', 3000, 'bond')])
def test_convolution_of_many_and_few_probabilities(gpu, kind, L, model, precision):
    """2, 4 or 8 (on the tensor cores 4, 8 or 32) probabilities per thread
    block: the same bits."""
    from pypercolate_gb300.ensemble import Ensemble
    got = []
    for P in (32, 1000, 5000):
        ps = np.concatenate([np.linspace(0.02, 0.97, 32), np.linspace(0.4, 0.6, P - 32)])
        e = Ensemble(kind, L, ps, precision=precision, model=model, window=0 if L != 24 else 200)
        e.run(130, key=3)
        assert e.errors() == 0
        got.append(e.mean.cpu().numpy().reshape(P, -1)[:32])
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize('kind,L,model,runs', [('grid', 24, 'bond', 130), ('torus', 20, 'site', 300),
                                               ('chain', 3000, 'bond', 5)])
def test_fp64_convolution_of_many_and_few_probabilities(gpu, kind, L, model, runs):
    from pypercolate_gb300.ensemble import Ensemble
    got = []
    for P in (16, 300, 5000):  # 2, 2 or 4, 8 probabilities per thread block
        ps = np.concatenate([np.linspace(0.02, 0.97, 16), np.linspace(0.4, 0.6, P - 16)])
        e = Ensemble(kind, L, ps, precision='fp64', model=model)
        e.run(runs, key=3)
        assert e.errors() == 0
        got.append(e.mean.cpu().numpy().reshape(P, -1)[:16])
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])

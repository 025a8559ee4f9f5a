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

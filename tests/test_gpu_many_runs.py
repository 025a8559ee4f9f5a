"""Launches of very many runs of small lattices: the paths taken there against
those of few runs, and against the oracle."""
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


def _micro(ens):
    return {k: v.cpu().numpy() for k, v in ens.micro.items()}


@pytest.mark.parametrize('kind,L,model,wrap', [
    ('grid', 2, 'bond', 'either'), ('grid', 9, 'bond', 'either'), ('grid', 16, 'bond', 'either'),
    ('chain', 33, 'bond', 'either'), ('grid', 16, 'site', 'either'), ('torus', 9, 'bond', 'x')])
@pytest.mark.parametrize('runs', [4096, 5001, 70001])
def test_sums_do_not_depend_on_the_slices(gpu, kind, L, model, wrap, runs):
    """One call, whose runs are reduced in slices, against calls of 2,047 runs,
    which are not: the exact sums are equal, and M2 is the pairwise merge."""
    from pypercolate_gb300.ensemble import Ensemble
    whole = Ensemble(kind, L, [0.5], model=model, wrap=wrap).run(runs, key=9)
    parts = Ensemble(kind, L, [0.5], model=model, wrap=wrap)
    for first in range(0, runs, 2047):
        parts.run(min(2047, runs - first), key=9, run0=first)
    a, b = _micro(whole), _micro(parts)
    for k in ('count', 'span_count', 'sum_lo', 'sum_hi'):
        assert np.array_equal(a[k], b[k]), k
    # M2 of one exact numerator against a merge of up to 35 parts, each of a few
    # roundings relative to the sum of squares
    sums = a['sum_lo'].view(np.uint64).astype(np.float64) + a['sum_hi'].astype(np.float64) * 2.0 ** 64
    np.testing.assert_allclose(a['m2'], b['m2'], rtol=1e-12, atol=1e-13 * (sums ** 2 / runs).max())
    assert whole.errors() == 0


# the smallest, the largest and odd sizes of the lattices whose node words lie in
# a block's shared memory with a thread per run (N <= 256, on the torus 121), and
# the first beyond
@pytest.mark.parametrize('kind,L,model,wrap', [
    ('grid', 1, 'bond', 'either'), ('grid', 2, 'bond', 'either'), ('grid', 9, 'bond', 'either'),
    ('grid', 16, 'bond', 'either'), ('grid', 17, 'bond', 'either'), ('chain', 1, 'bond', 'either'),
    ('chain', 2, 'bond', 'either'), ('chain', 256, 'bond', 'either'), ('chain', 257, 'bond', 'either'),
    ('torus', 1, 'bond', 'either'), ('torus', 2, 'bond', 'x'), ('torus', 3, 'bond', 'both'),
    ('torus', 11, 'bond', 'y'), ('torus', 12, 'bond', 'both'), ('grid', 1, 'site', 'either'),
    ('grid', 5, 'site', 'either'), ('grid', 16, 'site', 'either'), ('chain', 1, 'site', 'either'),
    ('chain', 173, 'site', 'either'), ('chain', 256, 'site', 'either'), ('torus', 1, 'site', 'either'), ('torus', 2, 'site', 'either'),
    ('torus', 7, 'site', 'both'), ('torus', 11, 'site', 'x')])
@pytest.mark.parametrize('window', [0, 37])
def test_ensembles_with_a_thread_per_run(gpu, kind, L, model, wrap, window):
    """40,001 runs at once (a thread each) and 20,000 and 20,001 (a block each)
    leave the same exact sums."""
    from pypercolate_gb300.ensemble import Ensemble
    whole = Ensemble(kind, L, [0.3, 0.6], model=model, wrap=wrap, window=window).run(40001, key=7, run0=5)
    parts = Ensemble(kind, L, [0.3, 0.6], model=model, wrap=wrap)
    parts.run(20000, key=7, run0=5)
    parts.run(20001, key=7, run0=20005)
    a, b = _micro(whole), _micro(parts)
    for k in ('count', 'span_count', 'sum_lo', 'sum_hi'):
        assert np.array_equal(a[k], b[k]), k
    assert whole.errors() == 0 and parts.errors() == 0
    # canonical means: FP32 sums of at most 400 rows, 2^-24 each
    np.testing.assert_allclose(whole.mean.cpu().numpy(), parts.mean.cpu().numpy(), rtol=3e-5, atol=1e-12)


def _planes(rec):
    """A record set's planes on the device, (rows, runs)."""
    return {k: getattr(rec, k)[:rec.rows * rec.n_runs].view(rec.rows, rec.n_runs)
            for k in ('max_span', 'm0', 'm2', 'm3', 'm4_lo', 'm4_hi', 'edge')}


def _same_as_in_parts(gpu, run, runs, part):
    """run(first, count)'s records at once and in parts of `part` runs."""
    import torch
    whole = _planes(run(0, runs))
    for first in range(0, runs, part):
        count = min(part, runs - first)
        few = _planes(run(first, count))
        for k, v in few.items():
            assert torch.equal(whole[k][:, first:first + count], v), (k, first)


@pytest.mark.parametrize('kind,L,model,wrap,runs', [
    ('grid', 1, 'bond', 'either', 40000), ('grid', 2, 'bond', 'either', 40000), ('grid', 11, 'bond', 'either', 40001),
    ('chain', 1, 'bond', 'either', 40000), ('chain', 70, 'bond', 'either', 40000),
    ('chain', 16385, 'bond', 'either', 24000), ('torus', 1, 'bond', 'either', 200000),
    ('torus', 2, 'bond', 'x', 200000), ('torus', 5, 'bond', 'both', 200001), ('torus', 129, 'bond', 'y', 16000),
    ('grid', 1, 'site', 'either', 200000), ('grid', 5, 'site', 'either', 200000),
    ('chain', 30, 'site', 'either', 200000)])
def test_records_with_a_thread_per_run(gpu, kind, L, model, wrap, runs):
    """n-major records of keyed permutations, a thread per run against a block
    per run."""
    from pypercolate_gb300 import hpc, lattice
    spec = lattice.lattice_spec(kind, L, model, wrap)
    _same_as_in_parts(gpu, lambda first, count: hpc._run_microcanonical(
        spec, True, rng='philox', key=29, run0=first, n_runs=count), runs, runs // 3 + 1)


@pytest.mark.parametrize('spanning', [True, False])
@pytest.mark.parametrize('both', [False, True])
def test_edge_lists_with_a_thread_per_run(gpu, oracle, spanning, both):
    """Given orders of self-loops, repeated edges and indices out of range,
    with and without a node on both sides."""
    from pypercolate_gb300 import hpc
    rng = np.random.default_rng(4)
    N, M, runs = 13, 30, 40000
    eu, ev = (rng.integers(0, N, M).astype(np.uint32) for _ in range(2))
    side = rng.choice([0, 0, 1, 2], N).astype(np.uint8)
    side[3] = 3 if both else 1
    spec = hpc.GraphSpec(gpu.GRAPH_EDGES, 0, N, M, eu, ev, side)
    perms = np.argsort(rng.random((runs, M)), axis=1).astype(np.uint32)
    perms[::5, 7] = M + 3
    _same_as_in_parts(gpu, lambda first, count: hpc._run_microcanonical(
        spec, spanning, perms=perms[first:first + count]), runs, runs // 3 + 1)
    host = hpc._run_microcanonical(spec, spanning, perms=perms).host()
    for r in (1, runs // 2 + 1, runs - 1):
        ref = oracle.sample_states(N, M, eu, ev, side, spanning, perms[r])
        assert np.array_equal(host['max_span'][:, r] & 0x7fffffff, ref['max'])
        assert np.array_equal(host['m2'][:, r], ref['moments_u64'][:, 2])
        if spanning:
            assert np.array_equal(host['max_span'][:, r] >> 31, ref['span'])


@pytest.mark.parametrize('kind,L,model', [
    ('chain', 501, 'bond'), ('chain', 502, 'site'), ('chain', 503, 'bond'), ('chain', 504, 'site'),
    ('grid', 23, 'bond'), ('grid', 25, 'site'), ('torus', 13, 'bond'), ('torus', 14, 'site')])
def test_node_words_between_windows(gpu, kind, L, model):
    """Places of runs at every multiple of 4 bytes, and copies that are no
    multiple of 16: the windows' sums are those of one window."""
    from pypercolate_gb300.ensemble import Ensemble
    a, b = (_micro(Ensemble(kind, L, [0.4], model=model, window=w).run(301, key=2)) for w in (0, 101))
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize('M', [1, 2, 3, 100, 255, 256])
@pytest.mark.parametrize('arrays', [False, True])
def test_short_permutations_of_many_seeds(gpu, M, arrays):
    """numpy's permutations of 32,768 seeds, a thread each, against those of
    fewer, a block each, and against numpy's own."""
    import torch
    rng = np.random.default_rng(M)
    runs, width = 32768, 3 if arrays else 1
    words = rng.integers(0, 2 ** 32, (runs, width), dtype=np.uint32)
    lens = rng.integers(1, width + 1, runs).astype(np.int32) if arrays else np.zeros(runs, np.int32)
    d_words, d_lens = gpu.to_device(words), gpu.to_device(lens)

    def draw(first, count):
        out = torch.empty(count * M, dtype=torch.int32, device='cuda')
        gpu.check(gpu.lib_handle().nz_permutations(
            M, count, gpu.PERM_MT19937, 0, 0, gpu.ptr(d_words[4 * width * first:]), gpu.ptr(d_lens[4 * first:]), width,
            gpu.ptr(out), gpu.stream_handle()), 'nz_permutations')
        return out.view(count, M)

    whole = draw(0, runs)
    for first in (0, 20000):
        assert torch.equal(whole[first:first + 12768], draw(first, 12768))
    for r in (0, 1, runs - 1):
        seed = words[r, :lens[r]].tolist() if arrays else int(words[r, 0])
        assert np.array_equal(whole[r].cpu().numpy(), np.random.RandomState(seed).permutation(M))


@pytest.mark.parametrize('runs,grid,chain,share,checkpoints', [
    (60000, (1, 16), (1, 64), 0.5, 256),           # more checkpoints than most have rows
    (130000, (8, 31), (64, 1000), 0.5, 64),        # all lattices up to 1,024 node words
    (60000, (33, 64), (2000, 4096), 0.1, 101),     # up to 4,096
    (50001, (64, 64), (64, 64), 0.0, 1000),        # one lattice
    (300000, (2, 90), (3, 9000), 0.4, 33)])        # some in blocks, some in threads
def test_fused_uneven_runs_in_threads(gpu, runs, grid, chain, share, checkpoints):
    """Every count, sum and M2 of the fused reduction of very many runs is that
    of the records', and of the fused one with too few node slots for threads."""
    from pypercolate_gb300.mix import MixEnsemble
    out = []
    for fused, threads in ((False, None), (True, None), (True, 8)):
        m = MixEnsemble(runs, grid=grid, chain=chain, chain_share=share, checkpoints=checkpoints, fused=fused,
                        threads=threads).run(77)
        out.append(m.results())
        del m
    for other in out[1:]:
        for k, v in out[0].items():
            assert np.array_equal(v, other[k]), k

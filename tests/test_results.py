"""The arrays that calls return belong to the caller alone."""
import numpy as np
import pytest

ROWS = ('microcanonical_statistics', 'canonical_statistics', 'canonical_averages', 'finalized_canonical_averages')


@pytest.mark.parametrize('name', ROWS)
@pytest.mark.parametrize('spanning', [True, False])
def test_row_types_are_not_shared(name, spanning):
    """Renaming the fields of one result leaves the next call's as they are."""
    from pypercolate_gb300 import hpc
    want = np.dtype(getattr(hpc, name + '_dtype')(spanning))
    rows = np.empty(3, dtype=hpc._dtype(name, spanning))
    assert rows.dtype == want
    rows.dtype.names = tuple('f%d' % i for i in range(len(want.names)))
    assert hpc._dtype(name, spanning).names == want.names


@pytest.mark.parametrize('spanning', [np.array(True), np.array(False), [0], [], {'a': 1}, np.True_, 1, None])
def test_row_types_of_any_truth_value(spanning):
    """As the types' own functions take it: by its truth, hashable or not."""
    from pypercolate_gb300 import hpc
    for name in ROWS:
        assert hpc._dtype(name, spanning) == np.dtype(getattr(hpc, name + '_dtype')(spanning))


@pytest.mark.gpu
@pytest.mark.parametrize('spanning', [True, False])
def test_rows_own_their_memory(spanning):
    """Rows can be resized in place, as arrays that are no views of others can."""
    torch = pytest.importorskip('torch')
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from pypercolate_gb300 import hpc, percolate
    from pypercolate_gb300.ensemble import Ensemble
    graph = percolate.percolation_graph(percolate.spanning_2d_grid(6), spanning_cluster=spanning)
    rows = hpc.bond_microcanonical_statistics(seed=1, **graph)
    stats = hpc.bond_canonical_statistics(rows, percolate.binomial_pmfs(graph['num_edges'], [0.2, 0.5]))
    averages = hpc.bond_initialize_canonical_averages(stats)
    ens = Ensemble('grid', 6, [0.4, 0.5], spanning=spanning).run(20, key=1)
    results = [rows, stats, averages, hpc.bond_reduce(averages, averages), ens.finalized(),
               hpc.finalize_canonical_averages(36, np.array([0.2, 0.5]), averages, 0.05)]
    del rows, stats, averages
    while results:
        a = results.pop()
        assert a.flags.owndata and a.flags.writeable
        a.resize(2 * a.shape[0])


@pytest.mark.gpu
def test_averages_share_nothing():
    """The arrays of one result do not overlap each other, nor those of the next."""
    torch = pytest.importorskip('torch')
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from pypercolate_gb300.ensemble import Ensemble
    ens = Ensemble('grid', 6, [0.4, 0.5]).run(20, key=1)
    arrays = [v for _ in range(2) for v in ens.microcanonical_averages().values() if isinstance(v, np.ndarray)]
    assert len(arrays) == 12
    for i, a in enumerate(arrays):
        assert a.flags.writeable and a.flags.c_contiguous
        assert not any(np.shares_memory(a, b) for b in arrays[:i])

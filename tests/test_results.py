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

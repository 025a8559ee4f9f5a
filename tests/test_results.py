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

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

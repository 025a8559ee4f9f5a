"""Sizes at which a launch's grid or a block's memory ends, on the GPU."""
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


# 262,136: the last number of probabilities whose tiles of 8, two blocks each,
# fit the grid's y; 524,280: the last that the entry point takes
@pytest.mark.parametrize('P', [262136, 262137, 300000, 524280])
@pytest.mark.parametrize('model', ['bond', 'site'])
def test_many_probabilities(gpu, P, model):
    """Every p of a long grid gets its canonical averages: those of the same
    values of p in an ensemble of few (same runs, same bits, whatever the
    tiles' probabilities)."""
    from pypercolate_gb300.ensemble import Ensemble
    ps = np.linspace(0.05, 0.95, P)
    ens = Ensemble('chain', 5, ps, precision='fp32', micro=False, model=model)
    ens.run(130, key=3)
    mean, m2 = (t.cpu().numpy().reshape(P, 7) for t in (ens.mean, ens.m2))
    for first in (0, P // 2 // 8 * 8, P - 16 - P % 8):
        few = Ensemble('chain', 5, ps[first:first + 16], precision='fp32', micro=False, model=model)
        few.run(130, key=3)
        for a, b in ((mean, few.mean), (m2, few.m2)):
            assert np.array_equal(a[first:first + 16], b.cpu().numpy().reshape(16, 7))

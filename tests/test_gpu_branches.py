"""Branches of dispatches that no other test reaches, against the oracle or
against the other branch."""
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


# tiles of 128 runs x 32 p: 13 x 2 = 26 (4 blocks to a tile, 8 for m4 with its high
# words), 50 x 2 = 100 (one, and 4)
@pytest.mark.parametrize('L,P', [(30, 400), (30, 1600), (340, 400), (340, 1600)])
def test_tensor_core_tiles_shared_by_4_and_8(gpu, L, P):
    """The bits of the canonical averages do not depend on how many blocks share
    a tile's probabilities: each 32 p by themselves are 2 tiles."""
    from pypercolate_gb300.ensemble import Ensemble
    ps = np.linspace(0.3, 0.7, P)
    whole = Ensemble('grid', L, ps, precision='tf32x3', micro=False).run(130, key=5)
    mean, m2 = (t.cpu().numpy().reshape(P, 7) for t in (whole.mean, whole.m2))
    assert whole.errors() == 0
    for first in {0, P // 2 // 32 * 32, (P - 1) // 32 * 32}:
        few = Ensemble('grid', L, ps[first:first + 32], precision='tf32x3', micro=False).run(130, key=5)
        for a, b in ((mean, few.mean), (m2, few.m2)):
            assert np.array_equal(a[first:first + 32], b.cpu().numpy().reshape(-1, 7))


# warps per run of few runs: 3, 6 and 8 in shared memory (an eighth of a run's bonds
# bounds a batch of 64 per warp); 12 in global memory, of more runs than SMs
@pytest.mark.parametrize('L,runs', [(30, 5), (40, 5), (50, 5), (257, 153)])
def test_records_of_other_warp_counts(gpu, oracle, L, runs):
    from pypercolate_gb300 import hpc
    spec = hpc.GraphSpec(gpu.GRAPH_GRID2D, L)
    rec = hpc._run_microcanonical(spec, True, rng='philox', key=17, run0=5, n_runs=runs)
    planes = {k: getattr(rec, k).view(spec.M + 1, runs) for k in ('max_span', 'm0', 'm2', 'm3', 'm4_lo')}
    for r in (0, runs - 1):
        ref = oracle.lattice_run(oracle.GRID_2D, L, oracle.philox_permutation(17, 5 + r, spec.M))
        got = {k: v[:, r].cpu().numpy() for k, v in planes.items()}
        ms = got['max_span'].view(np.uint32)
        assert np.array_equal(ms & 0x7fffffff, ref['max']) and np.array_equal(ms >> 31, ref['span'])
        for k, j in (('m0', 0), ('m2', 2), ('m3', 3), ('m4_lo', 4)):
            assert np.array_equal(got[k].astype(np.uint64) if k == 'm0' else got[k].view(np.uint64),
                                  ref['moments_u64'][:, j]), k

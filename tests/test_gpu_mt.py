"""numpy's permutations from the GPU: equal to RandomState's, element by
element, at the sizes where the draws' mask, the swaps' width and the place of
the shuffled array change."""
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


def _seeded(gpu, M, seeds):
    import torch
    from pypercolate_gb300 import hpc
    words = [hpc._mt_seed_words(s) for s in seeds]
    stride = max(len(w) for w, _ in words)
    flat = np.zeros((len(seeds), stride), np.uint32)
    lens = np.array([ln for _, ln in words], np.int32)
    for i, (w, _) in enumerate(words):
        flat[i, :len(w)] = w
    out = torch.empty(len(seeds) * M, dtype=torch.int32, device='cuda')
    gpu.check(gpu.lib_handle().nz_permutations(
        M, len(seeds), gpu.PERM_MT19937, 0, 0, gpu.ptr(gpu.to_device(flat)), gpu.ptr(gpu.to_device(lens)), stride,
        gpu.ptr(out), gpu.stream_handle()), 'nz_permutations')
    return out.cpu().numpy().reshape(len(seeds), M)


@pytest.mark.parametrize('M', [1, 2, 3, 31, 32, 33, 63, 64, 65, 480, 623, 624, 625, 1984, 4097, 65536, 65537, 100000])
def test_seeded(gpu, M):
    seeds = [0, 1, 12345, 2 ** 32 - 1, [1, 2, 3], list(range(700))]
    got = _seeded(gpu, M, seeds)
    for r, s in enumerate(seeds):
        assert np.array_equal(got[r], np.random.RandomState(s).permutation(M)), (M, s)


@pytest.mark.parametrize('M,runs', [(0, 2), (1, 3), (2, 700), (5, 100), (39, 16), (312, 5), (700, 4), (70000, 2)])
@pytest.mark.parametrize('drawn', [0, 1, 623, 624, 1000])
def test_global_stream(gpu, M, runs, drawn):
    """np.random's own stream, continued from any position and left where
    numpy would leave it."""
    from pypercolate_gb300 import percolate
    np.random.seed(99)
    np.random.randint(0, 2 ** 32, size=drawn, dtype=np.uint32) if drawn else None
    state = np.random.get_state()
    want = [np.random.permutation(M) for _ in range(runs)]
    after = np.random.get_state()
    np.random.set_state(state)
    got = percolate._global_stream_perms(M, runs).cpu().numpy()[:runs * M].reshape(runs, M)
    here = np.random.get_state()
    assert all(np.array_equal(g, w) for g, w in zip(got, want))
    assert here[2] == after[2] and np.array_equal(here[1], after[1])

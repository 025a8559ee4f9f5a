"""Memory that uneven batches ask for (no GPU needed: a size, not a call)."""
import pytest


@pytest.fixture(scope='module')
def lib():
    pytest.importorskip('torch')
    from pypercolate_gb300 import _native as nat
    from pypercolate_gb300 import build
    build.build()
    return nat


def _bytes(nat, runs, grid, chain, threads, fused, checkpoints=256):
    spec = nat.NzMixSpec()
    spec.grid_min, spec.grid_max = grid
    spec.chain_min, spec.chain_max = chain
    spec.chain_share, spec.checkpoints, spec.reduction = 1 << 31, checkpoints, int(fused)
    return nat.lib_handle().nz_mix_workspace_bytes(spec, runs, threads)


def test_node_slots_of_what_runs_at_a_time(lib):
    """Places for the 304 runs beyond shared memory that are resident at a time, or
    slots of 4,096 words for 116,736 threads, not one of the largest lattice's words
    for each of 49,152; and never more than the slots that are named."""
    runs, records = 100000, 36 * 256 * 100000
    small, place = 4 * 4096, 4 * 512 * 512
    default = _bytes(lib, runs, (8, 512), (1024, 65536), 49152, False)
    assert default < records + 100001 * small + (8 << 20)
    assert _bytes(lib, runs, (8, 512), (1024, 65536), 10, False) < records + 10 * place + (8 << 20)
    few = 36 * 256 * 10000
    assert 304 * place < _bytes(lib, 10000, (8, 512), (1024, 65536), 49152, False) - few < 304 * place + (8 << 20)
    assert _bytes(lib, 10000, (8, 256), (1024, 65536), 49152, False) < few + (8 << 20)
    threads = _bytes(lib, 10 ** 6, (8, 64), (1024, 4096), 10 ** 6, True)
    assert 116736 * small < threads < 116736 * small + (1 << 30)
    # all of the entry point's range still has a size
    for threads in (1, 304, 49152, 10 ** 6):
        for args in (((1, 1), (1, 1)), ((1, 1448), (1, 1 << 21))):
            for f in (False, True):
                assert _bytes(lib, 5, *args, threads, f, 2) > 0

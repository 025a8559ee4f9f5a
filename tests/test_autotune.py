"""What the tuners try and remember (no GPU needed)."""
import types

import pytest


def test_cached_choices_are_of_these_kernels(tmp_path, monkeypatch):
    """A choice made with other kernels is not found."""
    from pypercolate_gb300 import autotune as A
    monkeypatch.setattr(A.nat, 'torch_cuda', lambda: types.SimpleNamespace(
        cuda=types.SimpleNamespace(get_device_name=lambda: 'GPU')))
    keys = set()
    for i, source in enumerate(('a', 'b', 'a')):
        csrc = tmp_path / str(i)
        csrc.mkdir()
        (csrc / 'k.cu').write_text(source)
        monkeypatch.setattr(A, 'CSRC', str(csrc))
        keys.add(A._key(('mix2', 1)))
        assert A._key(('mix2', 1)) != A._key(('mix2', 2))
    assert len(keys) == 2 and 'GPU|mix2,1' not in keys


@pytest.mark.parametrize('M,runs', [(130560, 100000), (18624, 4000), (180, 10 ** 6)])
def test_ensemble_candidates_have_an_effect(M, runs):
    """Every candidate but the defaults changes a shape that a kernel depends on."""
    from pypercolate_gb300 import autotune as A
    first, *others = A.ensemble_candidates(M, runs)
    for c in others:
        changed = {k for k in c if c[k] != first[k]}
        assert changed and changed <= {'taper', 'window', 'reduce_slices'}


def test_one_shape_of_uneven_batches():
    """Slots, threads per CTA and shared-memory words are not timed: no launch
    depends on them."""
    from pypercolate_gb300 import autotune as A
    assert len(A._MIX_SHAPES) == 1 and A._MIX_SHAPES[0][0] >= 304


@pytest.mark.parametrize('grid,chain', [((2, 16), (2, 64)), ((8, 64), (64, 4096)), ((8, 512), (1024, 65536))])
@pytest.mark.parametrize('fused', [False, True])
def test_uneven_batches_are_tuned_with_all_node_words(grid, chain, fused):
    """The shape that is timed takes no slot from a batch of very many small
    lattices: as much memory as with a slot for every run."""
    pytest.importorskip('torch')
    from pypercolate_gb300 import _native as nat
    from pypercolate_gb300 import autotune as A
    from pypercolate_gb300 import build
    build.build()
    spec = nat.NzMixSpec()
    spec.grid_min, spec.grid_max = grid
    spec.chain_min, spec.chain_max = chain
    spec.chain_share, spec.checkpoints, spec.reduction = 1 << 31, 256, int(fused)
    size = nat.lib_handle().nz_mix_workspace_bytes
    assert size(spec, 10 ** 6, A._MIX_SHAPES[0][0]) == size(spec, 10 ** 6, 10 ** 6)

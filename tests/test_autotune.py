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

"""What the tuners try and remember (no GPU needed)."""
import types


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

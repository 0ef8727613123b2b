"""A host module (csrc/hkv_host.cpp) that is absent, does not load or belongs to another torch costs host time only: the
wrappers' Python path serves and checks every call, with one warning, and the next build replaces the module."""
import warnings

import pytest
import torch

from horizon_kernels_b200 import _lib, build
from horizon_kernels_b200 import kernels as K


@pytest.fixture
def unloaded(monkeypatch):
    build.build()
    monkeypatch.setattr(_lib, "_host", None)


def _calls():
    """each wrapper on CPU tensors: its Python path raises that there is no CPU path"""
    k = torch.zeros(2, 2, 128, dtype=torch.bfloat16)
    q = torch.zeros(2, 8, 128, dtype=torch.bfloat16)
    flat, st, g = tuple(torch.zeros(16, dtype=torch.uint8) for _ in range(4)), (1, 1, 1, 1, 1, 1), torch.ones(2)
    bt, lens, qsl = (torch.zeros(s, dtype=torch.int32) for s in ((2, 4), (2,), (3,)))
    for call in (lambda: K.write(k, k, flat, st, 16, torch.zeros(2, dtype=torch.int64), g, g),
                 lambda: K.decode_ragged(q, flat, st, 16, bt, lens, qsl, 1.0, 1.0, g, g, 1, q.clone(), flat[0]),
                 lambda: K.prefill(q, flat, st, 16, bt, [(0, 0, 2, 5)], 1.0, 1.0, 2, q.clone())):
        with pytest.raises(RuntimeError, match="no CPU path"):
            call()


def test_absent(unloaded, monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "HOST_PATH", str(tmp_path / "hkv_host.so"))
    with pytest.warns(RuntimeWarning, match="Python path") as w:
        _calls()
    assert len(w) == 1


def test_does_not_load(unloaded, monkeypatch, tmp_path):
    bad = tmp_path / "hkv_host.so"
    bad.write_bytes(b"not a library")
    monkeypatch.setattr(_lib, "HOST_PATH", str(bad))
    with pytest.warns(RuntimeWarning, match="Python path") as w:
        _calls()
    assert len(w) == 1


def test_another_torch(unloaded, monkeypatch):
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    with pytest.warns(RuntimeWarning, match="built for torch"):
        assert _lib.host().write() is None
    built = []
    monkeypatch.setattr(build, "build_host", lambda: built.append(1))
    build.build()
    assert built == [1]


def test_the_built_module_is_this_torch_s(unloaded, monkeypatch):
    monkeypatch.setattr(build, "build_host", lambda: pytest.fail("rebuilt"))
    build.build()
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _lib.host() is not _lib._NoHost


@pytest.mark.parametrize("missing", [n for n in vars(_lib._NoHost) if not n.startswith("_")] + ["bind"])
def test_a_module_of_an_older_source(unloaded, monkeypatch, tmp_path, missing):
    """built for this torch, before the source gained a function (libraries are not under version control, so a checkout that is brought
    up to date has one until the next build): the Python path serves, and the build replaces it"""
    old = tmp_path / "hkv_host.py"                   # (the loader goes by the suffix)
    names = [n for n in vars(_lib._NoHost) if not n.startswith("_")]
    old.write_text(f"torch_version = {str(torch.__version__)!r}\n" + "".join(
        f"def {n}(*a):\n    return None\n" for n in [*names, "bind"] if n != missing))
    monkeypatch.setattr(_lib, "HOST_PATH", str(old))
    with pytest.warns(RuntimeWarning, match="Python path") as w:
        _calls()
        assert _lib.host().layer_write() is None and _lib.host().layer_decode() is None
    assert len(w) == 1
    monkeypatch.setattr(build, "HOST", str(old))
    assert not build._host_loads()


def test_a_module_that_binds_other_entry_points(unloaded, monkeypatch, tmp_path):
    old = tmp_path / "hkv_host.py"
    old.write_text(f"torch_version = {str(torch.__version__)!r}\ndef bind(a, b):\n    pass\n" + "".join(
        f"def {n}(*a):\n    return None\n" for n in vars(_lib._NoHost) if not n.startswith("_")))
    monkeypatch.setattr(_lib, "HOST_PATH", str(old))
    with pytest.warns(RuntimeWarning, match="Python path"):
        _calls()

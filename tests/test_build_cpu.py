"""When the compiled parts are rebuilt."""
import os
import shutil

import pytest
import torch

import flash_attention_b200 as fa
from flash_attention_b200 import _lib


@pytest.fixture
def built(tmp_path, monkeypatch):
    """The installed extension and its record, as copies that a test may touch."""
    fa.build()
    for name in ("HOST_PATH", "HOST_ABI_PATH"):
        copy = str(tmp_path / os.path.basename(getattr(_lib, name)))
        shutil.copy2(getattr(_lib, name), copy)
        monkeypatch.setattr(_lib, name, copy)


def test_host_extension_is_rebuilt_for_another_torch(built, monkeypatch):
    assert not _lib._host_needs_build()
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert _lib._host_needs_build()


def test_host_extension_of_unknown_origin_is_rebuilt(built):
    os.unlink(_lib.HOST_ABI_PATH)
    assert _lib._host_needs_build()


def test_host_extension_of_another_torch_is_not_loaded(built, monkeypatch):
    """Without a compiler the stale extension is refused by name instead of being loaded."""
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(shutil, "which", lambda name: None)
    with pytest.raises(RuntimeError, match="built for another installation"):
        _lib.host()

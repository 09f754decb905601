"""The tuning cache's key holds the library: another build is tuned anew."""
import types

import pytest

from braids_hkt_gb300 import autotune


def test_key_changes_with_the_library(tmp_path, monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device: "a device")
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    library = tmp_path / "library.so"
    monkeypatch.setattr(autotune, "LIBRARY", library)
    s = types.SimpleNamespace(precision="mixed", method="fwave", nc=3, nf=7, nscen=1)
    keys = []
    for content in (b"one", b"two", b"one"):
        library.write_bytes(content)
        keys.append(autotune._key(s))
    assert keys[0] == keys[2] != keys[1]
    s.nc = 4
    assert autotune._key(s) != keys[2]
    library.unlink()
    with pytest.raises(FileNotFoundError):
        autotune._key(s)

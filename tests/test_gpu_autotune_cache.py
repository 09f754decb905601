"""A tuning cache that an earlier library left: its entries, which name the
gather's shape (kind 4, now part of the update), are not applied, and the
shape itself is accepted as before and changes no result."""
import json

import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_entry_of_an_earlier_library(precision, tmp_path, monkeypatch):
    import torch

    from braids_hkt_gb300 import autotune
    from braids_hkt_gb300.solver import RiverSolver
    case = S.small_channel()
    s, plain = RiverSolver(case, precision=precision), RiverSolver(case, precision=precision)
    store = tmp_path / "autotune.json"
    monkeypatch.setattr(autotune, "CACHE", store)
    device = torch.cuda.get_device_name(torch.cuda.current_device())
    key = f"{device}|{s.precision}|{s.method}|{s.nc}|{s.nf}|{s.nscen}"
    store.write_text(json.dumps({key: {"shapes": {"0": [256, 16], "4": [256, 32]}, "chunk": 8, "tile": None}}))
    assert not autotune.tune(s, reps=1, blocks=(128,), per_sm=(8,), chunks=(4,), tiles=())["cached"]
    again = autotune.tune(s, reps=1, blocks=(128,), per_sm=(8,), chunks=(4,), tiles=())
    assert again["cached"]
    s.set_launch_shape(4, 128, 8)
    assert s.launch_shape(4)[:2] == (128, 8)
    s.advance(0.5, 0.0)
    plain.advance(0.5, 0.0)
    np.testing.assert_array_equal(s.state(), plain.state())

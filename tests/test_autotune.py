"""The launch-shape autotuner's stored choices (host side)."""

import json

import pytest
import torch

from pyjuice_b200 import autotune
from pyjuice_b200.layer import layers as mod


@pytest.fixture
def tuner(monkeypatch):
    monkeypatch.delenv("PCB_AUTOTUNE_CACHE", raising=False)
    t = autotune.Autotuner()
    t.enabled = False  # no timing: the first candidate where nothing is stored
    return t


def test_a_stored_choice_is_one_of_the_candidates(tuner):
    """A choice kept by a call with more forms on offer is not taken by one that cannot run it, and
    stays with those that can."""
    tuner.choices["f|2|64"] = ("ws", 64)
    key = ("f", 2, 64)
    assert tuner.pick(key, [(32, 1), ("ws", 64)], None) == ("ws", 64)
    assert tuner.pick(key, [(32, 1), (64, 1)], None) == (32, 1)
    tuner.choices[tuner._key(("f|2|64", "among", (32, 1), (64, 1)))] = (64, 1)
    assert tuner.pick(key, [(32, 1), (64, 1)], None) == (64, 1)
    assert tuner.pick(key, [(32, 1), ("ws", 64)], None) == ("ws", 64)


def test_choices_from_a_file(tuner, tmp_path, monkeypatch):
    """Tuples come back from the file as what they were: a stored choice is still a candidate."""
    path = tmp_path / "choices.json"
    path.write_text(json.dumps({"f|1": ["tm", 0], "g|1": 32}))
    monkeypatch.setenv("PCB_AUTOTUNE_CACHE", str(path))
    t = autotune.Autotuner()
    t.enabled = False
    assert t.pick(("f", 1), [("tm", 1), ("tm", 0)], None) == ("tm", 0)
    assert t.pick(("g", 1), [16, 32], None) == 32


@pytest.mark.parametrize("run_rows,B,ld,prec", [(0, 64, 64, 2), (32, 63, 63, 2), (32, 64, 65, 2), (32, 64, 64, 3)])
def test_tma_form_only_where_it_runs(run_rows, B, ld, prec, monkeypatch):
    """A stored choice of the TMA form does not reach rows that it cannot read: chunks, blocks of
    other sizes (run_rows 0), unaligned rows, the E4M3 form."""
    names = []
    monkeypatch.setattr(mod.nat, "call", lambda name, *args: names.append(name))
    monkeypatch.setattr(mod.nat, "ptr", lambda t: None)
    monkeypatch.setattr(mod, "_num_sms", lambda: 148)
    monkeypatch.setattr(mod.TUNER, "enabled", False)
    monkeypatch.setattr(mod.TUNER, "choices", {f"tc05|0|{prec}|16|{B}": ("ws", 64)})
    rows = torch.zeros([64, ld])[:, :B]
    tiles = torch.zeros([16, 8], dtype=torch.int32)
    mod._tc05_call(rows, None, None, rows, ld, B, None, tiles, None, 0, prec, None, run_rows)
    assert names == ["pcb_lse_contract_tc05"]

"""The launch tuner's choice: the kernel's own chunk among the candidates, and
which saved tables stand."""

from __future__ import annotations

import json

import pytest
import torch

from gm1_b200.autotune import LEVEL_CHUNKS, Autotuner

pytestmark = pytest.mark.gpu


def _run(fastest, calls):
    def run(c):
        calls.append(c)
        torch.cuda._sleep(20_000 if c == fastest else 400_000)
    return run


@pytest.mark.parametrize("fastest", [0, 4, 64])
def test_the_fastest_is_chosen(fastest):
    tuner, calls = Autotuner(), []
    assert tuner.choose("kind", 640, 768, 80, _run(fastest, calls)) == fastest
    assert set(calls) == {c for c in LEVEL_CHUNKS if c <= 80}
    (entry,) = tuner.table.values()
    assert entry["chosen"] == fastest and entry["best"] != 0


def test_only_given_candidates_are_run():
    calls = []
    assert Autotuner().choose("kind", 8, 8, 40, _run(2, calls), candidates=(1, 2, 64)) == 2
    assert set(calls) == {1, 2}


def test_saved_tables(tmp_path):
    """A table this version saved is taken; one of earlier kernels (keys
    without their version) is searched again."""
    path, calls = tmp_path / "table.json", []
    tuner = Autotuner(path)
    assert tuner.choose("kind", 16, 12, 20, _run(8, calls)) == 8
    tuner.save()
    calls.clear()
    assert Autotuner(path).choose("kind", 16, 12, 20, _run(1, calls)) == 8 and calls == []
    path.write_text(json.dumps({"kind:16x12x20": {"best": 1, "ms": {"1": 0.1}}}))
    assert Autotuner(path).choose("kind", 16, 12, 20, _run(8, calls)) == 8 and calls != []

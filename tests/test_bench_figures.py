"""Figures of the bench line, on the CPU: the traversal form that it names."""
from __future__ import annotations

import sys

import pytest

from conftest import ROOT, mccfr

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402

L = mccfr.lib


@pytest.mark.parametrize("preset,changes,form", [
    (L.PRESET_6MAX_100BB, {}, "walk"),
    (L.PRESET_HU_20BB, {"raise_cap": 6}, "walk"),       # 28 decisions
    (L.PRESET_HU_20BB, {"raise_cap": 7}, "levels"),     # 32
    (L.PRESET_HU_20BB, {"raise_cap": 7, "max_depth": 31}, "walk"),
    (L.PRESET_HU_20BB, {"raise_cap": 0}, "levels"),     # as many as the depth cut allows
    (L.PRESET_HU_20BB, {"raise_cap": 0, "max_depth": 31}, "walk"),
    (L.PRESET_6MAX_100BB, {"traversal_form": L.FORM_LEVELS}, "levels"),
    (L.PRESET_6MAX_100BB, {"traversal_form": L.FORM_LANES}, "lanes"),
    (L.PRESET_REF8, {}, "reference"),
])
def test_traversal_form(preset, changes, form):
    cfg = L.preset(preset)
    for k, v in changes.items():
        setattr(cfg, k, v)
    assert bench.traversal_form(cfg) == form


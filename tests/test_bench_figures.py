"""Figures of the bench line, on the CPU: the traversal form that it names, and the
apply kernel's rate from one update's rows and the same update's time."""
from __future__ import annotations

import sys
from types import SimpleNamespace

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


def test_apply_rate_of_the_last_update():
    s0 = SimpleNamespace(apply_ms=0.0, last_apply_ms=9.0, touched_last=0, wide_rows_last=0)
    s1 = SimpleNamespace(apply_ms=8.0, last_apply_ms=2.5, touched_last=1_000_000, wide_rows_last=250_000)
    a = bench.apply_roofline(s0, s1, 4, 6000.0, row_bytes=192.0, wide_bytes=160.0, last=True)
    assert a["kernel_ms_per_launch"] == 2.5
    assert a["achieved"] == pytest.approx((1_000_000 * 192 + 250_000 * 160) / 0.0025 / 1e9)
    assert bench.apply_roofline(s0, s1, 4, 6000.0)["kernel_ms_per_launch"] == 2.0

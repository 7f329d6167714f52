"""Planes per block: the fused sweep's own default is not the staged sweeps'."""

from __future__ import annotations

import pytest
from default_engines import compiled_box, engine

pytestmark = pytest.mark.gpu


def test_default_fused_height_stays_with_the_fused_sweep() -> None:
    eng = engine(compiled_box((400, 388, 60)))  # tiles that nearly fill the chip: all planes
    fused = eng.get_tuning()
    assert fused[0] > 32 and fused[1] == 3
    eng.set_tuning(0, 2)
    assert eng.get_tuning() == (16, 2)
    eng.set_tuning(0, 3)
    assert eng.get_tuning() == fused
    eng.set_tuning(8, 3)  # the caller's height is everyone's
    assert eng.get_tuning() == (8, 3)
    eng.set_tuning(0, 2)
    assert eng.get_tuning() == (8, 2)
    eng.close()

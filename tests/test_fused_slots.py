"""The fused sweep's slot rings at every chunk height around their depth (4 E planes and 3 H planes are
staged when a march starts; shorter marches, one refill, several), against the oracle bit for bit."""

from __future__ import annotations

import pytest
from test_direct_sweeps import CPML, _model
from test_gpu_engine import check_against_oracles

from open_analysis_gb300.model import compile_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes", [1, 2, 3, 4, 5, 7])
@pytest.mark.parametrize("poles", [0, 1])
def test_fused_chunk_heights(planes: int, poles: int) -> None:
    from open_analysis_gb300.engine import Gb300Engine

    c = compile_model(_model((60, 46, 30), CPML, 4, poles), "float32")
    eng = Gb300Engine(c, "float32", max_steps=12)
    eng.set_tuning(planes, 3)
    eng.step(9)
    check_against_oracles(c, eng, 9, "float32")

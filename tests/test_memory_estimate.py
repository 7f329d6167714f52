"""The device bytes counted for a problem against what an engine at its defaults holds."""

from __future__ import annotations

import pytest

from open_analysis_gb300.model import compile_model
from open_analysis_gb300.structures import microstrip, via_transition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype, itemsize", [("float32", 4), ("float64", 8)])
@pytest.mark.parametrize("model", [lambda: microstrip(240, 120, 80), lambda: via_transition(161, 143, 88)])
def test_estimate_of_direct_sweep_grids(model, dtype: str, itemsize: int) -> None:  # type: ignore[no-untyped-def]
    """Grids that the direct sweeps run hold one set of fields."""
    from open_analysis_gb300.engine import Gb300Engine, estimate_bytes

    c = compile_model(model(), "float32")
    eng = Gb300Engine(c, dtype, max_steps=256)
    assert eng.get_tuning()[1] == 0
    peak = eng.peak_bytes()
    eng.close()
    est = estimate_bytes(c, itemsize, max_steps=256)
    assert peak <= est <= 1.1 * peak, (peak, est)

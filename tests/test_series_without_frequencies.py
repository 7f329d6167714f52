"""Recorded time series of a model without DFT frequencies: every step's sample is there."""

from __future__ import annotations

import numpy as np
import pytest
from test_direct_sweeps import CPML, _model

from open_analysis_gb300.model import compile_model
from oracle.numpy_engine import OracleEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("variant", [0, 2])
@pytest.mark.parametrize("batched", [False, True])
def test_series_without_frequencies_match_oracle(variant: int, dtype: str, batched: bool) -> None:
    """A captured chunk, remainders and single steps: the last sample of each comes from the launch
    that ends it. Float64 sums of the same samples: 1e-12 of their peak, as with frequencies."""
    from open_analysis_gb300.batch import EngineBatch
    from open_analysis_gb300.engine import Gb300Engine

    m = _model((26, 22, 20), CPML, n_freq=0, probes=3)
    m.conductors.clear()  # the copper fit needs frequencies
    c = compile_model(m, "float32")
    eng = Gb300Engine(c, dtype, record_series=True, max_steps=200)
    eng.set_tuning(8, variant)
    batch = EngineBatch([eng]) if batched else None
    for k in (64, 3, 1, 70):
        (batch or eng).step(k)
    ref = OracleEngine(c, dtype, record_series=True)
    ref.step(138)
    got, want = eng.series(), ref.series()
    assert set(got) == set(want)
    for name, v in want.items():
        assert np.abs(got[name] - v).max() <= 1e-12 * np.abs(v).max(), name
    assert all(v.size == 0 for v in eng.results().values())
    if batch is not None:
        batch.close()
    eng.close()

"""The surface impedance of one, two, four and other numbers of batch members, each precision, against
the oracle bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
from test_direct_sweeps import CPML, _model
from test_gpu_engine import check_against_oracles

from open_analysis_gb300.model import compile_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("members", [1, 2, 3, 4])
def test_sibc_of_every_member(members: int, dtype: str) -> None:
    from open_analysis_gb300.engine import Gb300Engine

    m = _model((44, 30, 20), CPML, 4, 0)
    m.drive = np.array([[1.0 - 0.3 * k, 0.5 * k] for k in range(members)])
    c = compile_model(m, "float32")
    assert c.sibc is not None and c.batch == members
    eng = Gb300Engine(c, dtype, max_steps=24)
    eng.step(20)
    check_against_oracles(c, eng, 20, dtype)

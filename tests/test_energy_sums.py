"""The energy sum's split of a grid over threads, against the oracle's float64 sum of the same fields."""

from __future__ import annotations

import numpy as np
import pytest
from test_direct_sweeps import CPML, _model

from open_analysis_gb300.model import compile_model
from oracle.numpy_engine import OracleEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
# fewer quads than a block has threads; two members meeting inside a block; several blocks; all blocks, many turns
@pytest.mark.parametrize("n", [(12, 9, 8), (30, 14, 12), (61, 50, 40), (250, 190, 120)])
def test_energy_of_random_fields(n: tuple[int, int, int], dtype: str) -> None:
    from open_analysis_gb300.engine import Gb300Engine

    c = compile_model(_model(n, CPML, 3), "float32")
    eng, ref = Gb300Engine(c, dtype), OracleEngine(c, dtype)
    rng = np.random.default_rng(sum(n))
    nx, ny, nz = c.grid.n
    for k in range(6):
        f = np.zeros((c.batch, *c.grid.shape), dtype)
        f[:, 1:nz, 1:ny, 1:nx] = rng.standard_normal((c.batch, nz - 1, ny - 1, nx - 1)) * 10.0 ** rng.integers(-9, 3)
        eng.set_field(k, f)
        (ref.E, ref.H)[k // 3][k % 3][...] = f
    # relative errors of positive sums: 2^-45 of a pair, 2^-53 times the turns and partial sums of
    # either side; together below 1e-12
    want = ref.energy()
    assert want > 0 and abs(eng.energy() - want) <= 1e-12 * want

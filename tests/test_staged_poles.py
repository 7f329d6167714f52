"""Several Debye poles in the staged and the fused sweeps."""

from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
from test_direct_sweeps import CPML, _model

from open_analysis_gb300.model import Region, compile_model
from oracle.numpy_engine import OracleEngine

pytestmark = pytest.mark.gpu
H = 0.2e-3


def _patchy(n, poles):  # type: ignore[no-untyped-def]
    """The dispersive slab with plain and conducting blocks cut into it at every offset within a quad."""
    m = _model(n, CPML, 4, poles, "dispersive")
    nx, ny, nz = n
    for k in range(6):
        x = 9 + 7 * k
        m.regions.append(Region((x * H, 6 * H, 3 * H), ((x + 1 + k % 3) * H, (8 + 2 * k) * H, (4 + k % 3) * H), 2.2, 0.02 * k))
    return compile_model(m, "float32")


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("poles", [2, 3, 5, 8])
def test_poles_in_staged_sweeps_match_oracle(poles: int, variant: int, dtype: str) -> None:
    """Quads of plain, dispersive and listed cells, from seeded fields: bit for bit."""
    from open_analysis_gb300.engine import Gb300Engine

    c = _patchy((61, 30, 22), poles)
    eng = Gb300Engine(c, dtype, max_steps=16)
    eng.set_tuning(5, variant)
    ref = OracleEngine(c, dtype, pole_sum="loop")
    rng = np.random.default_rng(31)
    for k, arr in enumerate(ref.E + ref.H):
        arr[...] = rng.standard_normal(arr.shape, dtype=np.float32)
        eng.set_field(k, arr)
    eng.step(4)
    ref.step(4)
    for k, want in enumerate(ref.E + ref.H):
        assert np.array_equal(eng.field(k), want.astype(np.float64)), k
    eng.close()


def test_five_poles_cost_the_fused_sweep_little_more_than_one() -> None:
    """A grid past the L2 cache with eight dispersive planes of a hundred: per cell and member 48 bytes of
    fields, 3 of indices and 24 per pole in eight cells of a hundred, so 61 bytes with five poles and 53 with
    one, a ratio of 1.15; a quarter more for their arithmetic."""
    from open_analysis_gb300.engine import Gb300Engine

    ms = []
    for poles in (1, 5):
        m = _model((400, 240, 100), CPML, 8, poles)
        m.regions[0] = replace(m.regions[0], hi=(1, 1, 10 * H))
        eng = Gb300Engine(compile_model(m, "float32"), "float32", max_steps=600)
        eng.set_tuning(16, 3)
        eng.step(64)
        ms.append(min(eng.step_timed(64) for _ in range(3)))
        eng.close()
    assert ms[1] <= 1.25 * 1.15 * ms[0], ms

"""CPML on grids so thin that the low and the high x slab share one vector of cells."""

from __future__ import annotations

import numpy as np
import pytest
from test_direct_sweeps import CPML, _model

from open_analysis_gb300.model import compile_model
from oracle.numpy_engine import OracleEngine

pytestmark = pytest.mark.gpu

# nx = 2 cells + 1 or + 2: the slabs' last and first cells lie in one four-cell vector (E and H at
# (9, 4), H alone at the others), or just not ((13, 5), (12, 5))
THIN = [((9, 12, 14), 4), ((10, 12, 14), 4), ((11, 13, 15), 5), ((17, 18, 19), 8), ((18, 19, 18), 8),
        ((13, 13, 14), 5), ((12, 13, 14), 5)]


def _seeded(c, dtype, eng):  # type: ignore[no-untyped-def]
    ref = OracleEngine(c, dtype, pole_sum="loop")
    rng = np.random.default_rng(23)
    for k, arr in enumerate(ref.E + ref.H):
        arr[...] = rng.standard_normal(arr.shape, dtype=np.float32)
        eng.set_field(k, arr)
    return ref


def _check(eng, ref) -> None:  # type: ignore[no-untyped-def]
    for k, want in enumerate(ref.E + ref.H):
        assert np.array_equal(eng.field(k), want.astype(np.float64)), k


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("variant", [0, 2])
@pytest.mark.parametrize("n, cells", THIN)
def test_thin_grid_matches_oracle(n, cells, variant, dtype) -> None:  # type: ignore[no-untyped-def]
    """From seeded fields, bit for bit; one pole and several (kernels of their own)."""
    from open_analysis_gb300.engine import Gb300Engine

    for poles in (1, 3):
        c = compile_model(_model(n, CPML, cells, poles), "float32")
        eng = Gb300Engine(c, dtype, max_steps=8)
        eng.set_tuning(8, variant)
        ref = _seeded(c, dtype, eng)
        eng.step(4)
        eng.half_h()
        eng.half_e()
        ref.step(5)
        _check(eng, ref)
        eng.close()


def test_thin_grids_in_a_batch_match_oracle() -> None:
    """Thin and ordinary grids, one and several poles, in the launches of one batch."""
    from open_analysis_gb300.batch import EngineBatch
    from open_analysis_gb300.engine import Gb300Engine

    engines, refs = [], []
    for n, cells, poles in [((9, 12, 14), 4, 1), ((30, 20, 18), 4, 1), ((17, 18, 19), 8, 2), ((26, 18, 19), 4, 2)]:
        c = compile_model(_model(n, CPML, cells, poles), "float32")
        engines.append(Gb300Engine(c, "float32", max_steps=80))
        refs.append(_seeded(c, "float32", engines[-1]))
    batch = EngineBatch(engines)
    batch.step(66)
    for e, ref in zip(engines, refs, strict=True):
        ref.step(66)
        _check(e, ref)
    batch.close()
    for e in engines:
        e.close()

"""Batches of engines whose current fields lie in the second buffers of the fused sweep."""

from __future__ import annotations

import numpy as np
import pytest
from default_engines import compiled_box, engine, seed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_engines_left_in_the_second_buffers_step_them(variant: int) -> None:
    """An odd number of fused steps, then an in-place variant: the fields stay in the buffers they are in.
    60 steps to the end of the chunk, a captured one, a remainder."""
    from open_analysis_gb300.batch import EngineBatch

    cs = [compiled_box((40, 36, 30)), compiled_box((52, 30, 28))]
    together, alone = [[engine(c) for c in cs] for _ in range(2)]
    for k, (a, b) in enumerate(zip(together, alone, strict=True)):
        for e in (a, b):
            seed(e, k)
            e.set_tuning(8, 3)
            e.step(3)
            e.set_tuning(8, variant)
    batch = EngineBatch(together)
    batch.step(61 + 64 + 5)
    batch.close()
    for a, b in zip(together, alone, strict=True):
        b.step(61 + 64 + 5)
        for comp in range(6):
            assert np.array_equal(a.field(comp), b.field(comp)), comp
        for key, v in b.results().items():
            assert np.array_equal(a.results()[key], v), key
        a.close()
        b.close()

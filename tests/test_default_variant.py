"""The sweep variant that an engine starts with."""

from __future__ import annotations

import pytest
from default_engines import compiled_box, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, dispersive, want", [
    ((400, 300, 90), False, 3),   # 10.8 million cells: few dispersive edges, nearly all in the fused box
    ((400, 300, 90), True, 0),
    ((400, 270, 90), False, 0),   # 9.7 million
    ((400, 340, 30), False, 3),   # 4.1 million, batch 4: 16.3 million, above every limit
    ((560, 540, 18), False, 0),   # 5.4 million, batch 2: 10.9 million, most of it in the outer layers
])
def test_default_variant(n, dispersive, want) -> None:  # type: ignore[no-untyped-def]
    batch = 4 if n == (400, 340, 30) else (1 if n[2] == 90 else 2)
    c = compiled_box(n, poles=((0.3, 4e-12),) if dispersive else (), batch=batch)
    eng = engine(c)
    assert c.batch == batch and eng.get_tuning()[1] == want
    eng.close()


def test_default_of_a_plain_grid_that_the_fused_sweep_cannot_take() -> None:
    """10.8 million cells with more materials than the fused sweep's table holds: the direct sweeps."""
    eng = engine(compiled_box((400, 300, 90), batch=1, materials=300))
    assert eng.get_tuning()[1] == 0
    eng.close()

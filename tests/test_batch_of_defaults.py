"""Engines at their default launch shape in one native batch, whatever their size."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
from default_engines import compiled_box, engine, seed

from open_analysis_gb300 import native
from open_analysis_gb300.model import ModelError


@pytest.fixture(scope="module")
def compiled():  # type: ignore[no-untyped-def]
    """Two members of 9.3 million cells (the fused sweep by default, tiles that nearly fill the chip)
    and a small grid (the direct sweeps)."""
    return [compiled_box((400, 388, 60)), compiled_box((40, 36, 30))]


class _Batch:
    """A native batch of the engines as they are."""

    def __init__(self, engines) -> None:  # type: ignore[no-untyped-def]
        self.lib = native.load()
        arr = (C.c_void_p * len(engines))(*[e._h.value for e in engines])
        self.h = C.c_void_p()
        native.check(self.lib.oafdtd_batch_create(arr, len(engines), C.byref(self.h)), "batch_create")

    def step(self, n: int) -> None:
        native.check(self.lib.oafdtd_batch_step_async(self.h, n), "step")
        native.check(self.lib.oafdtd_batch_wait(self.h), "wait")

    def graph_kernels(self) -> int:
        n = C.c_int64()
        native.check(self.lib.oafdtd_batch_graph_kernels(self.h, C.byref(n)), "graph_kernels")
        return int(n.value)

    def close(self) -> None:
        self.lib.oafdtd_batch_destroy(self.h)


@pytest.mark.gpu
def test_default_engines_on_both_sides_of_the_direct_size_form_one_batch(compiled) -> None:  # type: ignore[no-untyped-def]
    """Both have a fused box, so that their defaults differ by size alone. Three steps first: the
    fused engine's buffers are then swapped, the direct one's are not. Then 61 eager steps, a graph, 5 eager."""
    together, alone = [[engine(c) for c in compiled] for _ in range(2)]
    assert [e.get_tuning()[1] for e in together] == [3, 0]
    for k, (a, b) in enumerate(zip(together, alone, strict=True)):
        for e in (a, b):
            seed(e, k)
            e.step(3)
    batch = _Batch(together)
    batch.step(61 + 64 + 5)
    assert batch.graph_kernels() > 64
    for a, b in zip(together, alone, strict=True):
        b.step(61 + 40)
        b.step(29)
    with pytest.raises(ValueError):  # past max_steps: refused before any engine moves
        batch.step(100)
    assert {e.step_count for e in together} == {3 + 61 + 64 + 5}
    batch.close()
    for a, b in zip(together, alone, strict=True):
        for comp in range(6):
            assert np.array_equal(a.field(comp), b.field(comp)), comp
        for key, v in b.results().items():
            assert np.array_equal(a.results()[key], v), key
        a.close()
        b.close()


@pytest.mark.gpu
def test_a_variant_set_by_the_caller_still_holds_a_batch_to_it(compiled) -> None:  # type: ignore[no-untyped-def]
    small, other = engine(compiled[1]), engine(compiled[1])
    other.set_tuning(8, 2)
    with pytest.raises(ModelError):  # fused by size alone before the direct sweeps took small grids
        _Batch([small, other])
    small.set_tuning(8, 3)
    with pytest.raises(ModelError):
        _Batch([small, other])
    small.set_tuning(8, 2)
    small.step(1)
    with pytest.raises(ModelError):  # not at the same step
        _Batch([small, other])
    other.step(1)
    _Batch([small, other]).close()
    small.close()
    other.close()

"""Probes over planes and volumes: their samples and what they cost a step."""

from __future__ import annotations

import time

import numpy as np
import pytest
from test_direct_sweeps import CPML, _model

from open_analysis_gb300.model import Probe, compile_model
from open_analysis_gb300.structures import microstrip
from oracle.numpy_engine import OracleEngine

pytestmark = pytest.mark.gpu
H = 0.2e-3


@pytest.mark.parametrize("variant", [0, 2])
def test_large_probe_samples_match_oracle(variant: int) -> None:
    """1 to 5000 points (less than a round of a block's lanes, whole rounds, remainders) over a chunk, a
    remainder, single steps and half steps: float64 sums of the same terms in another order, each within
    5000 x 2^-53 of the sum of the terms' sizes, which 1e-10 of the peak covers here a thousand times over."""
    from open_analysis_gb300.batch import EngineBatch
    from open_analysis_gb300.engine import Gb300Engine

    m = _model((30, 28, 24), CPML)
    for k, (a, b, c) in enumerate([(1, 1, 1), (9, 3, 3), (5, 8, 16), (10, 25, 4), (1, 20, 21), (20, 25, 10), (17, 13, 19)]):
        lo, hi = (2 * H, 2 * H, 2 * H), ((1 + a) * H, (1 + b) * H, (1 + c) * H)
        m.probes.append(Probe(f"le{k}", "E", 1, lo, hi, "mean"))
        m.probes.append(Probe(f"lh{k}", "H", 0, lo, hi))
    comp = compile_model(m, "float32")
    sizes = [np.asarray(p["flat"]).size for p in comp.probes]
    assert min(sizes) < 128 and max(sizes) > 4096
    engines = [Gb300Engine(comp, "float32", record_series=True, max_steps=160) for _ in range(2)]
    for e in engines:
        e.set_tuning(8, variant)
    batch = EngineBatch(engines[1:])
    for k in (64, 5, 1):
        engines[0].step(k)
        batch.step(k)
    batch.close()
    for e in engines:
        e.half_h()
        e.half_e()
    ref = OracleEngine(comp, "float32", record_series=True)
    ref.step(71)
    for e in engines:
        got, want = e.series(), ref.series()
        for name, v in want.items():
            assert np.abs(got[name] - v).max() <= 1e-10 * np.abs(v).max(), name
        got, want = e.results(), ref.results()
        for name, v in want.items():
            assert np.abs(got[name] - v).max() <= 1e-9 * np.abs(v).max(), name
        e.close()


def test_single_steps_with_large_probes_cost_little_more_than_a_chunk() -> None:
    """Thirty E probes over whole planes: a step by itself, whose samples are all taken at its end, against
    a step of a chunk (and the 0.1 ms a call may take on the host)."""
    from open_analysis_gb300.engine import Gb300Engine

    h = 50e-6
    m = microstrip(200, 160, 80)
    for k in range(30):
        m.probes.append(Probe(f"e{k}", "E", 2, ((10 + k) * h, 2 * h, 2 * h), ((10 + k) * h, 158 * h, 78 * h)))
    eng = Gb300Engine(compile_model(m, "float32"), "float32", max_steps=1000)
    eng.step(128)

    def median(n: int) -> float:
        ts = []
        for _ in range(7):
            t = time.perf_counter()
            eng.step(n)
            ts.append((time.perf_counter() - t) / n)
        return float(np.median(ts))

    chunk, one = median(64), median(1)
    assert one <= 2 * chunk + 1e-4, (one, chunk)
    eng.close()

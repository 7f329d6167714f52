"""The direct sweeps (variant 0) and the per-chunk DFT against the oracle, at the sizes where they can
go wrong: one to sixteen planes a march, grids narrower than a block, no interior, thin z slabs,
PMC walls that meet, injection beside the sweep and by the edge pass, many probes.

Fields equal the oracle's bit for bit; DFTs to 1e-9 of their peak (float64 sums of the same samples
in another order)."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_engine import check_against_oracles

from open_analysis_gb300.grid import Grid, uniform_lines
from open_analysis_gb300.model import Conductor, LumpedPort, Model, Probe, Region, SoftSource, Waveform, compile_model
from open_analysis_gb300.pml import CpmlSpec
from oracle.numpy_engine import OracleEngine

pytestmark = pytest.mark.gpu
H = 0.2e-3


def _model(n, walls, cells=4, poles=0, source="plain", n_freq=3, probes=1):  # type: ignore[no-untyped-def]
    nx, ny, nz = n
    m = Model(Grid(*(uniform_lines(k, H) for k in n)), Waveform("gauss_mod", 10e9, 18e9),
              np.linspace(1e9, 19e9, n_freq), walls=walls, cpml=CpmlSpec(cells=cells))
    deb = tuple((0.3 / poles, 4e-12 * 3**p) for p in range(poles))
    m.regions.append(Region((-1, -1, 2 * H), (1, 1, (nz // 2) * H), 3.7, 0.01, False, deb))
    cu = (nx // 2 - 2, nx // 2 + 2)
    m.conductors.append(Conductor((cu[0] * H, -1, (nz // 2) * H), (cu[1] * H, 1, (nz // 2 + 1) * H), 5.8e7, 35e-6))
    at = {"plain": (nx // 3, ny // 2, nz // 2 + 2), "dispersive": (nx // 3, ny // 2, 3), "cpml": (2, ny // 2, 3)}[source]
    p = tuple(k * H for k in at)
    m.sources.append(SoftSource("s", 2, p, p))
    m.ports.append(LumpedPort("p", 1, (p[0] + 2 * H, p[1], p[2]), (p[0] + 2 * H, p[1] + 2 * H, p[2]), 50.0))
    m.drive = np.array([[1.0, 0.5], [0.0, -2.0]])
    rng = np.random.default_rng(3)
    for k in range(probes):
        q = tuple((int(rng.integers(1, d - 1))) * H for d in n)
        m.probes.append(Probe(f"e{k}", "E", k % 3, q, q))
        m.probes.append(Probe(f"h{k}", "H", k % 3, q, q))
    return m


CPML = ("cpml",) * 6
MIXED = ("pmc", "cpml", "pmc", "pmc", "cpml", "pmc")


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize(
    "n, walls, cells, poles, source",
    [
        ((13, 11, 10), CPML, 4, 1, "plain"),          # slabs almost everywhere
        ((30, 14, 12), ("pec",) * 6, 4, 0, "plain"),  # no slab at all
        ((33, 17, 19), MIXED, 4, 3, "dispersive"),    # PMC walls meet on edges and at a corner
        ((21, 18, 16), ("pmc",) * 6, 4, 1, "plain"),
        ((38, 20, 22), CPML, 6, 2, "cpml"),           # a source in a slab: the edge pass injects
        ((129, 62, 33), CPML, 5, 1, "dispersive"),    # two planes a march, odd extents
    ],
)
def test_direct_sweep_matches_oracle(n, walls, cells, poles, source, dtype) -> None:  # type: ignore[no-untyped-def]
    from open_analysis_gb300.engine import Gb300Engine

    c = compile_model(_model(n, walls, cells, poles, source), "float32")
    eng = Gb300Engine(c, dtype, max_steps=80)
    eng.set_tuning(16, 0)
    eng.step(70)  # one captured chunk and six eager steps
    check_against_oracles(c, eng, 70, dtype)


@pytest.mark.parametrize("n, cells, poles", [((123, 61, 47), 5, 1), ((200, 90, 52), 6, 2), ((210, 200, 118), 10, 1),
                                             ((300, 130, 9), 4, 1)])
def test_long_marches_match_oracle_from_random_fields(n, cells, poles) -> None:  # type: ignore[no-untyped-def]
    """4, 8 and 16 planes a march, and thin z slabs that hold the march to fewer, from seeded fields."""
    from open_analysis_gb300.engine import Gb300Engine

    c = compile_model(_model(n, CPML, cells, poles), "float32")
    eng = Gb300Engine(c, "float32", max_steps=8)
    eng.set_tuning(16, 0)
    ref = OracleEngine(c, "float32", pole_sum="loop")
    rng = np.random.default_rng(17)
    for k, arr in enumerate(ref.E + ref.H):
        arr[...] = rng.standard_normal(arr.shape, dtype=np.float32)
        eng.set_field(k, arr)
    eng.step(3)
    ref.step(3)
    for k, want in enumerate(ref.E + ref.H):
        assert np.array_equal(eng.field(k), want.astype(np.float64)), k


@pytest.mark.parametrize("n_freq, probes", [(1, 1), (5, 40), (257, 2)])
@pytest.mark.parametrize("variant", [0, 2])
def test_chunk_dft_matches_oracle(n_freq: int, probes: int, variant: int) -> None:
    """Running DFTs and recorded series over whole chunks, a remainder, single steps and half steps."""
    from open_analysis_gb300.engine import Gb300Engine

    c = compile_model(_model((26, 22, 20), CPML, n_freq=n_freq, probes=probes), "float32")
    eng = Gb300Engine(c, "float32", record_series=True, max_steps=200)
    eng.set_tuning(8, variant)
    ref = OracleEngine(c, "float32", record_series=True)
    for k in (64, 3, 1, 70):
        eng.step(k)
    eng.half_h()
    eng.half_e()
    ref.step(139)
    assert eng.step_count == 139
    got, want = eng.results(), ref.results()
    for name, v in want.items():
        assert np.abs(got[name] - v).max() <= 1e-9 * max(np.abs(v).max(), 1e-300), name
    for name, v in ref.series().items():
        assert np.abs(eng.series()[name] - v).max() <= 1e-12 * max(np.abs(v).max(), 1e-300), name

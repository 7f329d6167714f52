"""Problems and engines at their default launch shape, for the tests of the defaults."""

from __future__ import annotations

import numpy as np

from open_analysis_gb300.grid import Grid, uniform_lines
from open_analysis_gb300.model import Model, Probe, Region, SoftSource, Waveform, compile_model
from open_analysis_gb300.pml import CpmlSpec

H = 0.2e-3


def compiled_box(n, poles=(), batch=2, materials=0):  # type: ignore[no-untyped-def]
    nx, ny, nz = n
    m = Model(Grid(*(uniform_lines(k, H) for k in n)), Waveform("gauss_mod", 10e9, 18e9), np.linspace(1e9, 19e9, 3),
              walls=("cpml",) * 6, cpml=CpmlSpec(cells=6))
    m.regions.append(Region((-1, -1, 2 * H), (1, 1, (nz // 2) * H), 3.7, 0.01, False, poles))
    for k in range(materials):  # a row of little blocks, each of its own permittivity
        x, y = (8 + 3 * (k % 100)) * H, (8 + 3 * (k // 100)) * H
        m.regions.append(Region((x, y, (nz // 2) * H), (x + 2 * H, y + 2 * H, (nz // 2 + 2) * H), 1.5 + 0.01 * k))
    at = (nx // 3 * H, ny // 2 * H, (nz // 2 + 2) * H)
    m.sources.append(SoftSource("s", 2, at, at))
    m.probes.append(Probe("e", "E", 2, at, at))
    m.drive = np.linspace(1.0, -2.0, batch)[:, None]
    return compile_model(m, "float32")


def engine(c):  # type: ignore[no-untyped-def]
    from open_analysis_gb300.engine import Gb300Engine

    return Gb300Engine(c, "float32", max_steps=160)


def seed(eng, k: int) -> None:  # type: ignore[no-untyped-def]
    rng = np.random.default_rng(k)
    f = np.zeros(eng.field(0).shape)
    f[:, 8:-8, 8:-8, 8:28] = rng.standard_normal(f[:, 8:-8, 8:-8, 8:28].shape)
    eng.set_field(2, f)

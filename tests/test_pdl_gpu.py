"""Programmatic launches on and off give the same results bit for bit (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300.engine import DeviceSolver, make_plan, solve

pytestmark = pytest.mark.gpu


def _both(monkeypatch, call):
    out = []
    for value in ("1", "0"):  # read when a handle is created
        monkeypatch.setenv("CG_PDL", value)
        out.append(call())
    return out


# the second grid has the 2^20 cells from which y-passes are launched programmatically too
@pytest.mark.parametrize("shape,slabs", [((64, 96), 1), ((128, 96, 96), 1), ((45, 50, 45), 3)])
def test_solves(monkeypatch, shape, slabs):
    rng = np.random.default_rng(sum(shape))
    ids = rng.integers(0, 4, shape).astype(np.int32)
    med = cg.Medium.from_labels(ids, {i: (2.0 + i, 1000.0 + i, 1500.0 + 9 * i, 4.0) for i in range(4)})
    src = cg.CWSource(indices=np.array([[s // 2 for s in shape]], np.int64), phases=np.zeros(1, np.float32),
                      amplitude=8e5, f0=1e6)
    spec = cg.CWRunSpec(cfl=0.4, convergence_tol=0.0, min_settle_periods=2, max_settle_periods=3, n_record_periods=1)
    plan = make_plan("pdl", cg.Grid(shape, 0.2e-3, cg.PMLSpec(0.6e-3)), med, src, spec, nonlinear=True,
                     harmonics=(1, 2))

    def call():
        with DeviceSolver(plan, autotune=False) as dev:
            if slabs > 1:
                dev.set_slabs(slabs)
            return solve(plan, dev=dev)[0]

    a, b = _both(monkeypatch, call)
    for h in (1, 2):
        np.testing.assert_array_equal(a.phasors[h], b.phasors[h])
    np.testing.assert_array_equal(a.p_max, b.p_max)


@pytest.mark.parametrize("mode", ["labels", "dense"])
def test_heating(monkeypatch, mode):
    shape = (37, 45, 52)
    rng = np.random.default_rng(5)
    pick = rng.integers(0, 5, shape)
    maps = [(v[pick] if mode == "labels" else rng.uniform(v.min(), v.max(), shape)).astype(np.float32)
            for v in (rng.uniform(lo, hi, 5) for lo, hi in ((0.3, 0.6), (900, 1100), (3300, 3800), (0, 5e-3)))]
    q = (rng.random(shape) ** 3 * 4e6).astype(np.float32)
    t0 = (37.0 + rng.uniform(0, 8, shape)).astype(np.float32)

    def call():
        return cg.PennesSolverGB300().solve(t0, q, cg.ThermalMedium(*maps, dx=0.4e-3), dt=0.05, n_steps=40, dose=True)

    a, b = _both(monkeypatch, call)
    assert a.meta["coefficients"] == mode
    np.testing.assert_array_equal(a.temperature, b.temperature)
    np.testing.assert_array_equal(a.dose_cem43, b.dose_cem43)

"""Whole solves through the persistent z-passes of every kind against FP64 (GPU).

Drive, record window, convergence log and batch on three-level pencils (125,
243, 250, 375 points), 24- and 28-thread ones (384), bulk-copied and
per-thread field rows, and odd row counts, whose tiles are ragged.
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300.engine import DeviceSolver, make_plan, solve
from oracle import kspace as ok

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.complex128) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("shape,labelled,nonlinear,autotune", [
    ((6, 15, 125), True, True, False), ((6, 18, 125), False, False, False),
    ((6, 18, 243), False, True, False), ((6, 27, 243), True, False, False),
    ((6, 18, 250), True, True, False), ((5, 27, 250), False, True, False),
    ((5, 20, 375), True, False, False), ((6, 18, 384), True, True, False),
    ((6, 15, 384), False, False, False), ((6, 36, 384), True, False, True),
    ((9, 25, 96), True, True, False), ((8, 45, 160), False, True, True),
])
def test_a_batched_solve_matches_fp64(shape, labelled, nonlinear, autotune):
    rng = np.random.default_rng(sum(shape))
    dx = 0.25e-3
    lims = ((0.0, 20.0), (900.0, 1100.0), (1450.0, 1650.0), (3.0, 5.0) if nonlinear else (0.0, 0.0))
    if labelled:
        ids = rng.integers(0, 5, shape).astype(np.int32)
        vals = [rng.uniform(lo, hi, 5).astype(np.float32) for lo, hi in lims]
        med = cg.Medium.from_labels(ids, {i: tuple(float(v[i]) for v in vals) for i in range(5)})
        maps = [v[ids] for v in vals]
    else:
        maps = [rng.uniform(lo, hi, shape).astype(np.float32) for lo, hi in lims]
        med = cg.Medium(*maps)
    grid = cg.Grid(shape, dx, cg.PMLSpec(2 * dx))
    idx = np.array(sorted({tuple(int(rng.integers(2, s - 2)) for s in shape) for _ in range(20)}), np.int64)
    phases = rng.uniform(-np.pi, np.pi, (2, len(idx))).astype(np.float32)
    src = cg.CWSource(indices=idx, phases=phases[0], amplitude=5e5, f0=1e6)
    sched = dict(cfl=0.4, convergence_tol=0.0, min_settle_periods=2, max_settle_periods=3, n_record_periods=1)
    region = (slice(1, shape[0]), slice(2, shape[1] - 1), slice(3, shape[2] - 5))
    harmonics = (1, 2) if nonlinear else (1,)
    plan = make_plan("zpass", grid, med, src, cg.CWRunSpec(**sched), record_region=region, nonlinear=nonlinear,
                     harmonics=harmonics)
    with DeviceSolver(plan, batch=2, phases=phases, autotune=autotune) as dev:
        got = solve(plan, dev=dev, phases=phases)
    b = 1  # one member: the oracle takes seconds
    kw = dict(shape=shape, dx=dx, pml_vox_n=2, alpha=maps[0], rho=maps[1], c=maps[2], beta=maps[3], src_idx=idx,
              src_phase=phases[b], amplitude=5e5, f0=1e6, nonlinear=nonlinear, harmonics=harmonics,
              record_region=region, **sched)
    ref = ok.run_cw(**kw)
    assert got[b].steps_total == ref["steps_total"]
    for h in harmonics:
        # 1e-4, the phasor bound of the other solve tests, or twice what the float32 reference is
        # off by, where a weak harmonic makes that larger
        err = _rel(got[b].phasors[h], ref["phasors"][h])
        assert err < 1e-4 or err < 2.0 * _rel(ok.run_cw(**kw, dtype=np.float32)["phasors"][h], ref["phasors"][h])
    assert np.abs(got[b].p_max - ref["p_max"]).max() / np.abs(ref["p_max"]).max() < 1e-4
    np.testing.assert_allclose(np.array(got[b].convergence_history, np.float64).reshape(-1, 3)[:, 1],
                               np.array(ref["convergence_history"], np.float64).reshape(-1, 3)[:, 1], rtol=1e-4)

"""Phasors of a region that the sound has barely reached, against FP64 (GPU).

There the rounding of the transforms, of the loud part of the field, is what
shows. The bounds are 1.12 times the errors (relative L2) of transforms that
take the smaller factor of a pencil first, measured on these inputs.
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from oracle import kspace as ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,seed,measured", [
    ((24, 24, 192), 1, 3.120e-6), ((24, 24, 192), 2, 4.496e-6), ((24, 24, 192), 3, 3.320e-6),
    ((30, 30, 320), 1, 4.350e-6), ((30, 30, 320), 2, 5.139e-6), ((30, 30, 320), 3, 4.896e-6),
])
def test_quiet_phasors_are_as_close_to_fp64(shape, seed, measured):
    rng = np.random.default_rng(seed)
    dx = 0.25e-3
    grid = cg.Grid(shape, dx, cg.PMLSpec(6 * dx))
    ones = np.ones(shape, np.float32)
    med = cg.Medium(0.025 * ones, 1000 * ones, 1500 * ones, 0 * ones)
    idx = np.array(sorted({tuple(int(v) for v in (rng.integers(8, shape[0] - 8), rng.integers(8, shape[1] - 8), 12))
                           for _ in range(24)}), np.int64)
    phases = rng.uniform(-np.pi, np.pi, len(idx)).astype(np.float32)
    src = cg.CWSource(indices=idx, phases=phases, amplitude=1e5, f0=1e6, ramp_periods=3.0)
    sched = dict(convergence_tol=0.0, min_settle_periods=1, max_settle_periods=5, n_record_periods=1)
    region = tuple(slice(int(0.3 * n), int(0.7 * n)) for n in shape)
    ref_pt = tuple(int(v) for v in idx[0])
    res = cg.LinearKSpaceGB300().run(grid, med, src, cg.CWRunSpec(**sched), record_region=region,
                                     reference_point=ref_pt)
    ref = ok.run_cw(shape=shape, dx=dx, pml_vox_n=grid.pml_vox, alpha=med.alpha, rho=med.rho, c=med.c, beta=med.beta,
                    src_idx=idx, src_phase=phases, amplitude=1e5, f0=1e6, ramp_periods=3.0, nonlinear=False,
                    harmonics=(1,), record_region=region, reference_point=ref_pt, **sched)
    assert res.steps_total == ref["steps_total"]
    want = ref["phasors"][1]
    assert np.linalg.norm(res.phasors[1] - want) / np.linalg.norm(want) < 1.12 * measured

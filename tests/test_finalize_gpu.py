"""The phasors of a record window against their FP64 sums (GPU).

With one recorded period each phase bin holds exactly one pressure field, so
the phasors are 2/spp sum_n p_n exp(2 pi i h n / spp) of the fields the solver
hands out step by step. Amplitudes cover ordinary and huge fields, fields too
small for the kernel's float pairs, and cells that are exactly zero. (Fields too
large for the pairs overflow in the transforms before any phasor exists.)
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300 import engine as eng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-25, 1e-38, 1e24])
@pytest.mark.parametrize("harmonics", [(1,), (1, 2, 3), (1, 2, 3, 4, 5, 6, 7, 8)])
def test_phasors_are_the_fp64_sums_of_the_recorded_fields(harmonics, scale):
    shape = (5, 9, 24)
    rng = np.random.default_rng(3)
    ones = np.ones(shape, np.float32)
    med = cg.Medium(2.0 * ones, 1000.0 * ones, 1500.0 * ones, 0.0 * ones)
    grid = cg.Grid(shape, 0.1e-3, cg.PMLSpec(2 * 0.1e-3))
    src = cg.CWSource(indices=np.array([[2, 4, 12]], np.int64), phases=np.zeros(1, np.float32),
                      amplitude=1e-3 * scale, f0=1e6)
    spec = cg.CWRunSpec(cfl=0.3, convergence_tol=0.0, min_settle_periods=1, max_settle_periods=1, n_record_periods=1)
    plan = eng.make_plan("fin", grid, med, src, spec, harmonics=harmonics)
    p0 = (rng.standard_normal(shape) * 1e5 * scale).astype(np.float32)
    p0[:, 3] = 0.0
    u0 = np.zeros((3, 1, plan.ncell), np.float32)
    with eng.DeviceSolver(plan, autotune=False) as dev:
        dev.set_state(p0.reshape(1, -1), u0, 0)
        dev.begin_record()
        fields = []
        for _ in range(plan.spp):
            dev.run_steps(1, record=True)
            fields.append(dev.get_state()[0][0].reshape(shape).astype(np.float64))
        ph, pm = dev.finalize(plan.spp)
    fields = np.array(fields)
    assert np.isfinite(fields).all()
    np.testing.assert_array_equal(pm[0].reshape(shape), np.abs(fields).max(axis=0).astype(np.float32))
    n = np.arange(plan.spp)
    top = np.abs(fields).max()
    for i, h in enumerate(harmonics):
        want = np.tensordot(2.0 / plan.spp * np.exp(2j * np.pi * h * n / plan.spp), fields, axes=(0, 0))
        got = ph[0, i].reshape(shape)
        for a, b in ((got.real, want.real), (got.imag, want.imag)):
            # the final rounding to float32 (one spacing) and the sums' own error, below
            # 2^-44 of the largest term a step: 2^-40 of the largest field covers spp of them
            assert (np.abs(a - b) <= np.spacing(np.abs(b).astype(np.float32)) + 2.0**-40 * top).all()

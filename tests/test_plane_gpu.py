"""2-D grids, whose transverse chains run in one launch each (GPU).

Row lengths on every thread split of the y kernels, one without a kernel of
its own, row counts around a CTA's four or eight rows, batches, and restored
states.
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300 import engine as eng
from oracle import kspace as ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(36, 8), (64, 14), (45, 36), (96, 64), (125, 75), (180, 16), (320, 24), (384, 10),
                                   (512, 12), (9, 24), (405, 16)])
@pytest.mark.parametrize("batch", [1, 3])
def test_a_2d_step_matches_the_oracle_and_restores_bitwise(shape, batch):
    rng = np.random.default_rng(sum(shape))
    med = cg.Medium(*(rng.uniform(lo, hi, shape).astype(np.float32)
                      for lo, hi in ((0, 40), (900, 1100), (1450, 1650), (4, 5))))
    grid = cg.Grid(shape, 0.25e-3, cg.PMLSpec(2 * 0.25e-3))
    src = cg.CWSource(indices=np.array([[s // 2 for s in shape]], np.int64), phases=np.zeros(1, np.float32),
                      amplitude=1e5, f0=1e6)
    plan = eng.make_plan("plane", grid, med, src, cg.CWRunSpec(cfl=0.3), nonlinear=True)
    p0 = (rng.standard_normal((batch, plan.ncell)) * 1e5).astype(np.float32)
    u0 = (rng.standard_normal((3, batch, plan.ncell)) * 0.05).astype(np.float32)
    with eng.DeviceSolver(plan, batch=batch, autotune=False) as dev:
        dev.set_state(p0, u0, 0)
        dev.run_steps(1)  # the source ramp is zero at t = 0
        p1, u1 = dev.get_state()
        dev.run_steps(4)
        p5, u5 = dev.get_state()
        dev.set_state(p1, u1, 1)
        dev.run_steps(4)
        pr, ur = dev.get_state()
        bad = p0.copy()
        ubad = u0.copy()
        ubad[0, 0, 3] = np.nan  # the component across the plane
        dev.set_state(bad, ubad, 0)
        dev.run_steps(1)
        assert np.isnan(dev.get_state()[0][0]).any()  # 0 x NaN reaches the pressure, as the product with k_x = 0 does
    np.testing.assert_array_equal(p5, pr)
    np.testing.assert_array_equal(u5, ur)
    maps = ok.medium_maps(med.alpha, med.rho, med.c, med.beta, plan.padded, plan.dt, True, np.float64)
    ks = ok.k_vectors(plan.padded, plan.dx, np.float64)
    kap = ok.kappa_sinc(ks, plan.c_max, plan.dt, np.float64)
    der = ok.spectral_derivative_factors(ks, kap, plan.padded, np.complex128)
    spg = ok.sponge_volume(plan.padded, grid.pml_vox, 2.0, np.float64)
    for b in range(batch):
        want_p, want_u = ok.step_fields(p=p0[b].reshape(plan.padded).astype(np.float64),
                                        u=[u0[i, b].reshape(plan.padded).astype(np.float64) for i in (1, 2)],
                                        dt_over_rho=maps[0], rhoc2_dt=maps[1], absorb=maps[2], beta2_dt=maps[3],
                                        sponge=spg, deriv=der, padded=plan.padded)
        # 2e-6: the bound of the 3-D step tests
        assert np.abs(p1[b].reshape(plan.padded) - want_p).max() / np.abs(want_p).max() < 2e-6
        for i in range(2):
            assert np.abs(u1[1 + i, b].reshape(plan.padded) - want_u[i]).max() / np.abs(want_u[i]).max() < 2e-6

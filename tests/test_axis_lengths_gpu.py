"""Every size-specialised axis length against FP64 (GPU): transforms, one step, restored states.

The lengths are the 2/3/5-smooth ones from 36 to 400 that have kernels of
their own; each is put on the x, the y and the z axis, the last with an even
and an odd row count and row counts around one tile (16 or 32 rows), so that
ragged tiles, single last rows and label rows of every alignment occur.
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300 import engine as eng
from caustica_gb300.fft import FFT3D
from oracle import kspace as ok

pytestmark = pytest.mark.gpu

LENGTHS = [36, 40, 45, 50, 54, 60, 72, 75, 80, 81, 90, 100, 108, 120, 125, 135, 144, 150, 162, 180, 200, 216, 225,
           240, 243, 250, 270, 288, 300, 324, 360, 375, 384]


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", LENGTHS)
def test_transforms_match_numpy_fp64(n):
    # float32 butterflies over log2 n <= 9 levels: below 3e-6, the bound of the other lengths
    for shape in ((n, 3, 10), (3, n, 10), (2, 18, n), (2, 15, n), (1, 1, n)):
        rng = np.random.default_rng(n)
        x = rng.standard_normal((2, *shape)).astype(np.float32)
        with FFT3D(shape, batch=2) as f:
            spec = f.forward(x)
            back = f.inverse(spec) / np.prod(shape)
        want = np.fft.rfftn(x.astype(np.float64), axes=(1, 2, 3))
        assert _rel(FFT3D.to_numpy_layout(spec), want) < 3e-6, shape
        assert _rel(back, x) < 3e-6, shape


def _plan(shape, labelled, seed):
    rng = np.random.default_rng(seed)
    if labelled:
        ids = rng.integers(0, 5, shape).astype(np.int32)
        rows = {i: (float(rng.uniform(0, 40)), float(rng.uniform(900, 1100)), float(rng.uniform(1450, 1650)), 4.5)
                for i in range(5)}
        med = cg.Medium.from_labels(ids, rows)
    else:
        med = cg.Medium(*(rng.uniform(lo, hi, shape).astype(np.float32)
                          for lo, hi in ((0, 40), (900, 1100), (1450, 1650), (4, 5))))
    grid = cg.Grid(shape, 0.25e-3, cg.PMLSpec(2 * 0.25e-3))
    src = cg.CWSource(indices=np.array([[s // 2 for s in shape]], np.int64), phases=np.zeros(1, np.float32),
                      amplitude=1e5, f0=1e6)
    return eng.make_plan("len", grid, med, src, cg.CWRunSpec(cfl=0.3), nonlinear=True), grid, med, rng


STEPS = ([((4, 18, n), True) for n in (36, 75, 100, 125, 162, 240, 288, 375, 384)]
         + [((4, 17, n), lab) for n, lab in ((45, True), (81, False), (135, True), (150, True), (225, False),
                                             (250, True), (300, True), (320, False), (512, True), (640, True))]
         + [((n, 9, 16), True) for n in (45, 144, 300, 375)] + [((5, n, 16), True) for n in (54, 125, 180, 360)]
         + [((6, 33, 64), True), ((6, 15, 96), False)])


@pytest.mark.parametrize("shape,labelled", STEPS)
def test_a_step_matches_the_oracle_and_a_restored_state_continues_bitwise(shape, labelled):
    plan, grid, med, rng = _plan(shape, labelled, sum(shape))
    p0 = (rng.standard_normal(plan.padded) * 1e5).astype(np.float32)
    u0 = (rng.standard_normal((3, 1, plan.ncell)) * 0.05).astype(np.float32)
    with eng.DeviceSolver(plan, autotune=False) as dev:
        dev.set_state(p0.reshape(1, -1), u0, 0)
        dev.run_steps(1)  # the source ramp is zero at t = 0
        p1, u1 = dev.get_state()
        dev.run_steps(3)
        p4, u4 = dev.get_state()
        dev.set_state(p1, u1, 1)
        dev.run_steps(3)
        pr4, ur4 = dev.get_state()
    np.testing.assert_array_equal(p4, pr4)
    np.testing.assert_array_equal(u4, ur4)
    maps = ok.medium_maps(med.alpha, med.rho, med.c, med.beta, plan.padded, plan.dt, True, np.float64)
    ks = ok.k_vectors(plan.padded, plan.dx, np.float64)
    kap = ok.kappa_sinc(ks, plan.c_max, plan.dt, np.float64)
    der = ok.spectral_derivative_factors(ks, kap, plan.padded, np.complex128)
    spg = ok.sponge_volume(plan.padded, grid.pml_vox, 2.0, np.float64)
    pr, ur = ok.step_fields(p=p0.astype(np.float64), u=[u0[i, 0].reshape(plan.padded).astype(np.float64) for i in range(3)],
                            dt_over_rho=maps[0], rhoc2_dt=maps[1], absorb=maps[2], beta2_dt=maps[3], sponge=spg,
                            deriv=der, padded=plan.padded)
    # 2e-6: the bound of the other lengths' step test
    assert np.abs(p1[0].reshape(plan.padded) - pr).max() / np.abs(pr).max() < 2e-6
    for i in range(3):
        assert np.abs(u1[i, 0].reshape(plan.padded) - ur[i]).max() / np.abs(ur[i]).max() < 2e-6

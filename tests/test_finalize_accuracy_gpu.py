"""Phasors of sums that cancel, against exact arithmetic (GPU).

Each member holds a uniform pressure: it stays what it is up to the rounding of
the transforms, so a harmonic is what is left of terms 10^13 times larger, and
the error of the sum itself shows.
"""

from __future__ import annotations

from decimal import Decimal, getcontext

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300 import engine as eng

pytestmark = pytest.mark.gpu


def _cos_sin(num: int, den: int):
    """cos and sin of 2 pi num / den to 40 digits."""
    pi = Decimal("3.14159265358979323846264338327950288419716939937510")
    x = 2 * pi * num / den
    c, s, term = Decimal(0), Decimal(0), Decimal(1)
    for n in range(120):
        c, s = (c + term * (1 if n % 4 == 0 else -1), s) if n % 2 == 0 else (c, s + term * (1 if n % 4 == 1 else -1))
        term = term * x / (n + 1)
    return c, s


def test_cancelling_harmonics_are_as_accurate_as_fp64_sums():
    getcontext().prec = 45
    shape, batch, harmonics = (4, 6, 16), 24, (1, 2, 3)
    rng = np.random.default_rng(11)
    ones = np.ones(shape, np.float32)
    c = ones.copy()  # a slow medium with one fast voxel, which sets the time step
    c[0, 0, 0] = 1500.0
    med = cg.Medium(0.0 * ones, 1000.0 * ones, c, 0.0 * ones)
    grid = cg.Grid(shape, 0.25e-3, cg.PMLSpec(0.0))
    src = cg.CWSource(indices=np.array([[0, 0, 0]], np.int64), phases=np.zeros(1, np.float32), amplitude=1e-30, f0=1e6)
    spec = cg.CWRunSpec(cfl=0.48, convergence_tol=0.0, min_settle_periods=1, max_settle_periods=1, n_record_periods=1)
    plan = eng.make_plan("fin", grid, med, src, spec, harmonics=harmonics)
    amp = rng.uniform(1e5, 2e5, batch).astype(np.float32)
    p0 = np.repeat(amp[:, None], plan.ncell, 1)
    with eng.DeviceSolver(plan, batch=batch, autotune=False) as dev:
        dev.set_state(p0, np.zeros((3, batch, plan.ncell), np.float32), 0)
        dev.begin_record()
        fields = []
        for _ in range(plan.spp):
            dev.run_steps(1, record=True)
            fields.append(dev.get_state()[0][:, -1])  # the last voxel of each member
        ph = dev.finalize(plan.spp)[0].reshape(batch, len(harmonics), -1)[:, :, -1]
    fields = np.array(fields)
    assert plan.spp >= 5 and np.abs(fields / amp - 1).max() < 1e-5
    cs = [_cos_sin(n, plan.spp) for n in range(plan.spp)]
    for b in range(batch):
        for i, h in enumerate(harmonics):
            want = [sum(Decimal(float(fields[n, b])) * cs[h * n % plan.spp][j] for n in range(plan.spp)) * 2 / plan.spp
                    for j in range(2)]
            for got, w in ((ph[b, i].real, want[0]), (ph[b, i].imag, want[1])):
                # the FP64 factors, 1 ulp of the cosine and half a one of 2/spp each, come to 2^-51.3
                # of the field; one spacing of the result for the rounding to float32
                tol = 2.0**-50 * float(amp[b]) + float(np.spacing(np.abs(np.float32(w))))
                assert abs(float(Decimal(float(got)) - w)) <= tol, (b, h)

"""Pennes steps on per-cell coefficient maps against the reference's float32 path (GPU).

Sizes around the kernel's tile: one warp is 32 cells of a z row, a block eight
rows, and it walks eight or sixteen x planes; 2-D grids are one x plane.
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from oracle import pennes as op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 9, 8), (11, 3, 31), (9, 8, 32), (6, 9, 33), (17, 7, 65), (33, 2, 64), (2, 17, 97),
                                   (290, 2, 2), (13, 40), (40, 9)])
@pytest.mark.parametrize("boundary,tref,perfused", [("insulated", None, True), ("dirichlet", 36.0, True),
                                                    ("dirichlet", None, False)])
def test_dense_maps_equal_the_reference_float32_path(shape, boundary, tref, perfused):
    rng = np.random.default_rng(sum(shape))
    k = rng.uniform(0.3, 0.6, shape).astype(np.float32)
    rho = rng.uniform(900, 1100, shape).astype(np.float32)
    cp = rng.uniform(3300, 3800, shape).astype(np.float32)
    w = (rng.uniform(0, 5e-3, shape) if perfused else np.zeros(shape)).astype(np.float32)
    tm = cg.ThermalMedium(k, rho, cp, w, dx=0.4e-3)
    q = (rng.random(shape) ** 3 * 4e6).astype(np.float32)
    t0 = (37.0 + rng.uniform(0, 8, shape)).astype(np.float32)
    s = cg.PennesSolverGB300(boundary=boundary, reference_temperature_c=tref, on_unstable="substep")
    kw = dict(k=k, rho=rho, specific_heat=cp, perfusion=w, dx=tm.dx, dt=0.05, n_steps=23, boundary=boundary,
              reference_temperature_c=tref, on_unstable="substep")
    for dose, source in ((True, q), (False, None)):
        res = s.solve(t0, source, tm, dt=0.05, n_steps=23, dose=dose)
        assert res.meta["coefficients"] == "dense"
        ref = op.solve(t0, source, dtype=np.float32, dose=dose, **kw)
        np.testing.assert_array_equal(res.temperature, ref["temperature"])
        np.testing.assert_array_equal(res.temperature_max, ref["temperature_max"])
        if dose:
            ref64 = op.solve(t0, source, dtype=np.float64, dose=True, **kw)
            rel = np.abs(res.dose_cem43 - ref64["dose_cem43"]) / np.abs(ref64["dose_cem43"])
            assert rel.max() < 1e-3  # the bound of the label kernels' dose test

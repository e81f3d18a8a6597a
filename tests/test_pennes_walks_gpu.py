"""Pennes blocks that walk many x planes, against the reference's float32 path (GPU).

Grids whose tile counts make a block walk four or eight planes, the last run
ragged, and grids longer than one block dimension at eight planes a block.
"""

from __future__ import annotations

import numpy as np
import pytest

import caustica_gb300 as cg
from oracle import pennes as op

pytestmark = pytest.mark.gpu


def _check(shape, mode, boundary, n_steps, dose):
    rng = np.random.default_rng(sum(shape))
    if mode == "dense":
        k, rho, cp, w = (rng.uniform(lo, hi, shape).astype(np.float32)
                         for lo, hi in ((0.3, 0.6), (900, 1100), (3300, 3800), (0, 5e-3)))
    else:
        ids = rng.integers(0, 5, shape)
        k, rho, cp, w = (rng.uniform(lo, hi, 5).astype(np.float32)[ids]
                         for lo, hi in ((0.3, 0.6), (900, 1100), (3300, 3800), (0, 5e-3)))
    tm = cg.ThermalMedium(k, rho, cp, w, dx=0.4e-3)
    q = (rng.random(shape) ** 3 * 4e6).astype(np.float32)
    t0 = (37.0 + rng.uniform(0, 8, shape)).astype(np.float32)
    s = cg.PennesSolverGB300(boundary=boundary, reference_temperature_c=36.0, on_unstable="substep")
    res = s.solve(t0, q, tm, dt=0.05, n_steps=n_steps, dose=dose)
    assert res.meta["coefficients"] == mode
    kw = dict(k=k, rho=rho, specific_heat=cp, perfusion=w, dx=tm.dx, dt=0.05, n_steps=n_steps, boundary=boundary,
              reference_temperature_c=36.0, on_unstable="substep", dose=dose)
    ref = op.solve(t0, q, dtype=np.float32, **kw)
    np.testing.assert_array_equal(res.temperature, ref["temperature"])
    np.testing.assert_array_equal(res.temperature_max, ref["temperature_max"])
    if dose:
        want = op.solve(t0, q, dtype=np.float64, **kw)["dose_cem43"]
        assert (np.abs(res.dose_cem43 - want) / np.abs(want)).max() < 1e-3  # the bound of the other dose tests


@pytest.mark.parametrize("shape", [(524328, 2, 2), (524328, 2, 3)])  # z-pairs and single cells
@pytest.mark.parametrize("mode", ["labels", "dense"])
def test_grids_longer_than_one_block_dimension(shape, mode):
    _check(shape, mode, "insulated", 2, False)


@pytest.mark.parametrize("boundary,dose", [("insulated", True), ("dirichlet", False)])
@pytest.mark.parametrize("shape,mode", [
    ((37, 130, 131), "dense"),   # 85 tiles: four planes
    ((37, 180, 190), "dense"),   # 138 tiles: eight planes
    ((37, 130, 131), "labels"),  # single cells
    ((37, 180, 191), "labels"),
    ((37, 180, 190), "labels"),  # z-pairs, 72 tiles: four planes
    ((37, 290, 190), "labels"),  # 114 tiles: eight planes
])
def test_blocks_that_walk_four_and_eight_planes(shape, mode, boundary, dose):
    _check(shape, mode, boundary, 7, dose)

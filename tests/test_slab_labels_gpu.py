"""Slab mode on planes that do not start on a label word: bit-identical to the plain step (GPU).

A slab's labels start at its first plane. With ny = 2 mod 4 and an odd nz,
odd planes start two bytes into a 4-byte word, and a grid of odd nx ends two
bytes into one.
"""

from __future__ import annotations

import numpy as np
import pytest

from test_slabs_gpu import _case, _same, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,nonlinear,dense,slabs", [
    ((50, 50, 45), True, False, 2),   # second slab at plane 25
    ((45, 50, 45), False, False, 3),  # slabs at 15 and 30, last word of the volume not whole
    ((36, 54, 75), True, False, 4),   # slabs at 9, 18 and 27
    ((45, 90, 81), False, False, 2),  # even plane, last word not whole
    ((50, 50, 45), True, True, 2),
])
def test_slabs_that_start_inside_a_label_word(shape, nonlinear, dense, slabs):
    plan = _case(shape, nonlinear, seed=sum(shape) + slabs, dense=dense)
    _same(_solve(plan, 1)[0], _solve(plan, slabs)[0])


def test_batched_members_of_such_slabs():
    plan = _case((45, 50, 45), False, seed=21)
    phases = np.random.default_rng(4).uniform(-np.pi, np.pi, (2, plan.src_xyz.shape[0])).astype(np.float32)
    for a, b in zip(_solve(plan, 1, phases), _solve(plan, 3, phases)):
        _same(a, b)

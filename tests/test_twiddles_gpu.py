"""Twiddle factors of the transforms are the floats nearest to their values (GPU).

The transform of a unit impulse at element s of an axis is exp(-2 pi i s k / n);
its first few bins are table entries, read through codelets that only add zeros.
"""

from __future__ import annotations

import numpy as np
import pytest

from caustica_gb300.fft import FFT3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 128, 160, 192, 225, 256, 300, 320, 400, 512, 640])
@pytest.mark.parametrize("axis", [0, 1])
def test_an_impulse_transforms_to_the_nearest_floats(n, axis):
    shape = [2, 2, 2]
    shape[axis] = n
    with FFT3D(tuple(shape)) as f:
        for s in (1, 2, 3, 4):
            x = np.zeros((1, *shape), np.float32)
            x[(0, *(s if d == axis else 0 for d in range(3)))] = 1.0
            spec = np.moveaxis(FFT3D.to_numpy_layout(f.forward(x))[0], axis, 0)[:, 0, 0]
            for k in (1, 2, 3, 4):
                w = 2.0 * np.pi * s * k / n
                assert (spec[k].real, spec[k].imag) == (np.float32(np.cos(w)), np.float32(-np.sin(w))), (s, k)

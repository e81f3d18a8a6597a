"""The 3-D transform on the caller's device buffers (GPU).

Aligned, disjoint device buffers are transformed where they are; misaligned or
overlapping ones and host buffers go through the handle's staging arrays. Every
route gives the values of the host call bit for bit and leaves its input alone.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from caustica_gb300 import _lib
from caustica_gb300.fft import FFT3D

pytestmark = pytest.mark.gpu

# all axes on codelets, odd ny, an axis on the runtime-plan passes, 1-D
SHAPES = [(12, 16, 24), (9, 15, 36), (6, 8, 18), (405, 4, 8), (1, 1, 96)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("spec_offset", [0, 2, 4])  # floats: 16-, 8- and 16-byte aligned starts
@pytest.mark.parametrize("real_offset", [0, 1])
def test_device_buffers_give_the_host_call_bitwise(shape, spec_offset, real_offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((2, *shape)).astype(np.float32)
    with FFT3D(shape, batch=2) as f:
        spec = f.forward(x)
        back = f.inverse(spec)
        ns, nr = spec.size * 2, x.size
        xd = torch.zeros(nr + 8, device="cuda")
        xd[real_offset:real_offset + nr] = torch.from_numpy(x).cuda().reshape(-1)
        sd = torch.zeros(ns + 8, device="cuda")
        bd = torch.full((nr + 8,), 7.0, device="cuda")
        torch.cuda.synchronize()
        p = lambda t, off: C.c_void_p(t.data_ptr() + 4 * off)  # noqa: E731
        _lib.call("cg_fft3d_forward", f.h, p(xd, real_offset), p(sd, spec_offset))
        np.testing.assert_array_equal(sd[spec_offset:spec_offset + ns].cpu().numpy().view(np.complex64),
                                      spec.reshape(-1))
        np.testing.assert_array_equal(xd[real_offset:real_offset + nr].cpu().numpy(), x.reshape(-1))
        _lib.call("cg_fft3d_inverse", f.h, p(sd, spec_offset), p(bd, real_offset))
        np.testing.assert_array_equal(bd[real_offset:real_offset + nr].cpu().numpy(), back.reshape(-1))
        np.testing.assert_array_equal(sd[spec_offset:spec_offset + ns].cpu().numpy().view(np.complex64),
                                      spec.reshape(-1))
        assert float(bd[real_offset + nr:].min()) == 7.0 and float(sd[spec_offset + ns:].abs().max()) == 0.0


@pytest.mark.parametrize("shape", [(12, 16, 24), (9, 15, 36)])
def test_a_transform_may_overwrite_its_own_input(shape):
    torch = pytest.importorskip("torch")
    x = np.random.default_rng(1).standard_normal((1, *shape)).astype(np.float32)
    with FFT3D(shape) as f:
        spec = f.forward(x)
        back = f.inverse(spec)
        buf = torch.zeros(spec.size * 2, device="cuda")
        buf[:x.size] = torch.from_numpy(x).cuda().reshape(-1)
        torch.cuda.synchronize()
        _lib.call("cg_fft3d_forward", f.h, C.c_void_p(buf.data_ptr()), C.c_void_p(buf.data_ptr()))
        np.testing.assert_array_equal(buf.cpu().numpy().view(np.complex64), spec.reshape(-1))
        _lib.call("cg_fft3d_inverse", f.h, C.c_void_p(buf.data_ptr()), C.c_void_p(buf.data_ptr()))
        np.testing.assert_array_equal(buf[:x.size].cpu().numpy(), back.reshape(-1))

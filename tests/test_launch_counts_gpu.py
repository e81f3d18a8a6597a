"""Kernel launches that a handle reports and makes, counted by the profiler (GPU)."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import caustica_gb300 as cg
from caustica_gb300 import _lib
from caustica_gb300 import engine as eng

pytestmark = pytest.mark.gpu


def _solver(shape):
    rng = np.random.default_rng(sum(shape))
    ids = rng.integers(0, 3, shape).astype(np.int32)
    med = cg.Medium.from_labels(ids, {i: (2.0 + i, 1000.0 + i, 1500.0 + i, 0.0) for i in range(3)})
    grid = cg.Grid(shape, 0.25e-3, cg.PMLSpec(2 * 0.25e-3))
    src = cg.CWSource(indices=np.array([[s // 2 for s in shape]], np.int64), phases=np.zeros(1, np.float32),
                      amplitude=1e5, f0=1e6)
    return eng.DeviceSolver(eng.make_plan("launches", grid, med, src, cg.CWRunSpec(cfl=0.3)), autotune=False)


def _profiled(torch, call):
    """Names of the kernels, and of the runtime calls, that `call` makes."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU,
                                            torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    events = list(prof.events())
    kernels = [e.name for e in events if e.device_type == torch.autograd.DeviceType.CUDA]
    return kernels, [e.name for e in events if e.device_type == torch.autograd.DeviceType.CPU]


@pytest.fixture(scope="module")
def torch():
    """torch, with the profiler brought up: a process's first session sees no kernels."""
    torch = pytest.importorskip("torch")
    _profiled(torch, lambda: torch.zeros(1, device="cuda"))
    return torch


@pytest.mark.parametrize("shape,slabs,launches", [
    ((64, 96), 1, 4),       # one x plane: a transverse chain is one launch
    ((405, 16), 1, 8),      # one x plane, a row length without kernels of its own
    ((24, 32, 48), 1, 8),
    ((24, 32, 48), 3, 20),
])
def test_a_step_makes_the_launches_that_the_handle_reports(torch, shape, slabs, launches):
    with _solver(shape) as dev:
        if slabs > 1:
            dev.set_slabs(slabs)
        assert dev.launches_per_step == dev.config()["launches_per_step"] == launches
        dev.run_steps(2)

        def steps():
            dev.run_steps(5)
            dev.synchronize()

        kernels = [k for k in _profiled(torch, steps)[0] if "pass" in k or "plane" in k]
        assert len(kernels) == 5 * launches


@pytest.mark.parametrize("warmup", [0, 1])
def test_a_run_timed_by_graph_times_graph_launches_only(torch, warmup):
    with _solver((64, 96)) as dev:
        dev.run_periods(warmup)  # one period: plain launches, no graph yet
        ms = C.c_float()

        def timed():
            _lib.call("cg_solver_timed_run", dev.h, 2 * dev.plan.spp, 0, 1, C.byref(ms))

        calls = _profiled(torch, timed)[1]
        first = calls.index("cudaEventRecord")
        last = len(calls) - 1 - calls[::-1].index("cudaEventRecord")
        assert calls[first + 1:last] == ["cudaGraphLaunch"] * 2

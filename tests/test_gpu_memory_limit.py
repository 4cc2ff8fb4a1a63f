"""Grids that fit the device only without what the faster routes add (a second
buffer set in 2-D, padded rows in 3-D, a spare set where a later allocation
needs the room) still run, on the slower routes and to the same accuracy.  The
device's memory is taken up by one tensor but for a stated amount."""
import contextlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _Leave:
    """Leaves `mb` megabytes of device memory free (to about 2 MB)."""

    def __init__(self, mb):
        torch.cuda.init()
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        self.held = []
        free = torch.cuda.mem_get_info(0)[0]
        for unit in (1 << 30, 64 * MB, 2 * MB):
            while free - mb * MB >= unit:
                n = (free - mb * MB) // unit * unit
                try:
                    self.held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
                free = torch.cuda.mem_get_info(0)[0]

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.held.clear()
        torch.cuda.empty_cache()


@pytest.fixture
def warm(fdtd):
    with fdtd.Simulation(mode=2, size=(40, 40), precision=1) as s:   # the library's device code is loaded
        s.step(10)
        s.sync()
    with fdtd.Simulation(mode=3, size=(40, 40, 40), precision=1) as s:
        s.step(10)
        s.sync()
    return fdtd


# 4096^2 FP32 with PML: a set is 6 x 64 = 384 MB, the staging grid 128 MB.
# 1100: all fits; 850: both sets do, the staging grid takes the spare one's
# place; 560: one set and the staging grid
@pytest.mark.parametrize("mb", [1100, 850, 560])
@pytest.mark.parametrize("steps_first", [0, 7, 14])
def test_2d_without_room_for_a_second_set(warm, mb, steps_first):
    fdtd = warm
    kw = dict(mode=2, size=(4096, 4096), precision=1, use_pml=True, pml=8, point_source=(2048, 2048), point_source_mask=4)
    with fdtd.Simulation(**kw) as sim:
        sim.step(steps_first + 21)
        want = sim.field("Ez").copy()
    with _Leave(mb), fdtd.Simulation(**kw) as sim:
        sim.step(steps_first)
        before = sim.launch_count()
        sim.step(14)
        tiles = sim.launch_count() - before <= 3
        assert tiles == (mb > 600), sim.launch_count() - before
        first = sim.field("Ez").copy()
        before = sim.launch_count()
        sim.step(7)
        assert (sim.launch_count() - before <= 1) == (mb > 1000), sim.launch_count() - before
        got = sim.field("Ez")
    assert np.any(first != 0) and np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


# FP16 rows of 33 cells pad to 40.  PML: two sets of 36 B a cell are 363 MB, padded
# 439, the staging grid 40.  470: padded rows would leave no room for the staging
# grid and an eps map; 420: nor for themselves
@pytest.mark.parametrize("mb", [470, 420])
def test_3d_without_room_for_padded_rows(warm, mb):
    fdtd = warm
    n = (400, 400, 33)
    kw = dict(mode=3, size=n, precision=2, use_pml=True, pml=6)
    rng = np.random.default_rng(2)
    fields = {}
    for c in ("Ex", "Hz"):
        fields[c] = np.zeros(n)
        fields[c][1:-1, 1:-1, 1:-1] = rng.standard_normal([v - 2 for v in n]) / (1 if c[0] == "E" else 376.73)
    out = []
    for limit in (None, mb):
        with _Leave(limit) if limit else contextlib.nullcontext(), fdtd.Simulation(**kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.step(5, t_start=50)
            assert (sim.step_kernel == "fused3d_regblock") == bool(limit), sim.step_kernel
            out.append({c: sim.field(c) for c in fields})
    for c in fields:   # (five steps rounded to 11 bits, in pairs or singly)
        assert np.linalg.norm(out[1][c] - out[0][c]) <= 5e-3 * np.linalg.norm(out[0][c]), c

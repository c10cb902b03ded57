"""Scenes stepped without reading: the caller queues steps ahead of the GPU
where no window could be outgrown meanwhile, and no window clamps where one
could (a plain scene and a batch)."""

import copy
import time

import numpy as np
import pytest

from pfsim import _native as N
from pfsim import recipe as R
from pfsim import workloads as W

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def tank_at_rest(substeps):
    """A fluid that fills its tank from wall to wall, in a window that fits
    the tank: its spread stays as it is."""
    r = W.dam_break(20000, seed=31, substeps=substeps)
    s = 2.0 * r.radius
    pts = W.fill_box((-0.5, 0.0, -0.3), (0.5, 0.2, 0.3), s).astype(np.float32)
    n = len(pts)
    o = copy.deepcopy(r.materials[0][1])
    o.range = (0, n)
    r.capacity, r.uploads, r.materials = n, [R.Upload(0, pts)], [("fluid", o)]
    h = o.smoothing_radius
    r.loop.grid_min, r.loop.grid_max = (-0.5 - h, -h, -0.3 - h), (0.5 + h, 0.25, 0.3 + h)
    return r


@pytest.mark.parametrize("batch", [False, True])
def test_fluid_held_by_walls_queues_ahead(batch):
    """Three steps are queued in less host time than the GPU takes for one: a
    caller that waited for the step before each would need two of them."""
    r = tank_at_rest(substeps=40)
    s = R.NativeBackend().build(r)
    w = R.Batch([s]) if batch else s
    read = (lambda: w.readback(0, N.PF_FIELD_POSITIONS)) if batch else (lambda: w.readback(N.PF_FIELD_POSITIONS))
    for _ in range(20):
        w.step(DT)
    read()
    host, gpu = [], []
    for _ in range(5):
        t0 = time.perf_counter()
        for _ in range(3):
            w.step(DT)
        host.append(1e3 * (time.perf_counter() - t0))
        read()
        gpu.append(w.last_step_ms())
    print(f"three steps queued in {min(host):.3f} ms, one takes {min(gpu):.3f} ms")
    assert min(host) < min(gpu), (host, gpu)
    assert not (w.overflow(0) if batch else w.overflow())["grid_clamped"]


@pytest.mark.parametrize("scenes", [1, 6])
@pytest.mark.parametrize("batch", [False, True])
def test_close_window_never_clamps(monkeypatch, scenes, batch):
    """Dam breaks whose windows hold little more than their block, 60 steps
    without a read: no clamp, and the bits of the same scenes in windows that
    they never outgrow."""
    if scenes > 1 and not batch:
        pytest.skip("a plain scene is one scene")
    monkeypatch.setenv("PFSIM_NBR_PATH", "0")  # the other path agrees within tolerance only
    small, big = [], []
    for k in range(scenes):
        r = W.dam_break(20000 if scenes == 1 else 4000, seed=25 + k)
        h = r.materials[0][1].smoothing_radius
        r.loop.grid_min = (-0.5 - 2 * h, -2 * h, -0.3 - 2 * h)
        q = copy.deepcopy(r)
        r.loop.grid_max = (-0.1 + 2 * h, 0.5 + 2 * h, 0.3 + 2 * h)
        q.loop.grid_max = (0.5 + 2 * h, 12.0, 0.3 + 2 * h)
        small.append(r)
        big.append(q)
    out = []
    for recs in (small, big):
        built = [R.NativeBackend().build(r) for r in recs]
        w = R.Batch(built) if batch else built[0]
        for _ in range(60):
            w.step(DT)
        for i in range(scenes):
            assert not (w.overflow(i) if batch else w.overflow())["grid_clamped"], i
        out.append([w.readback(i, N.PF_FIELD_POSITIONS) if batch else w.readback(N.PF_FIELD_POSITIONS)
                    for i in range(scenes)])
        w.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)

"""A batch or field tuned by its autotuner is not slower than one left alone:
few small fields run on strips of one row, which no selectable shape has, and
what distinguishes the shapes there is less than a launch takes on the host."""
import time

import numpy as np
import pytest

from dim2d_finite_volume_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[128], [64, 100, 150]])
def test_tuned_batch_not_slower(sizes):
    """Steps of tuned and untuned batches in turn, medians of 15 runs of 64 steps;
    at most 1.1 times (1.2 and more where the autotuner leaves strips by size)."""
    from dim2d_finite_volume_b200 import batch, field
    batches, fields = {}, []
    for tuned in (False, True):
        bt = batches[tuned] = batch.Batch()
        for n in sizes:
            d = workloads.domain(n, n, T0=0.95, bubbles=[(0.0, 0.0, 0.15)], mach=0.0,
                                 bc="periodic_xy", li=0.2)
            f = field.Field(d["nx"], d["ny"], bc="periodic_xy")
            f.ini(d["nodes"], d["x_map"], d["y_map"])
            bt.add(f, 0.01 * d["dt"])
            fields.append(f)
        if tuned:
            shapes, times = bt.autotune()
            assert times[0][shapes[0]] == times[0].min()
        for _ in range(6):  # its graphs
            bt.step(64)
        bt.sync()
    times = {False: [], True: []}
    for _ in range(15):
        for tuned, bt in batches.items():
            t0 = time.perf_counter()
            bt.step(64)
            bt.sync()
            times[tuned].append(time.perf_counter() - t0)
    for bt in batches.values():
        bt.close()
    for f in fields:
        f.close()
    median = {tuned: np.median(ts) for tuned, ts in times.items()}
    assert median[True] <= 1.1 * median[False], median


@pytest.mark.parametrize("preset,n,ny", [("periodic_xy", 126, 130), ("reflection_xy", 66, 62),
                                         ("hedstrom_xy", 62, 66)])
def test_tuned_field_not_slower(preset, n, ny):
    """The same for a field against its default variant."""
    from dim2d_finite_volume_b200 import field
    d = workloads.domain(n, ny, T0=0.95, bubbles=[(0.0, 0.0, 0.15)], mach=0.0, bc=preset, li=0.2)
    fields = {}
    for tuned in (False, True):
        f = fields[tuned] = field.Field(d["nx"], d["ny"], bc=preset)
        f.ini(d["nodes"], d["x_map"], d["y_map"])
        if tuned:
            f.autotune()
    times = {False: [], True: []}
    for _ in range(17):
        for tuned, f in fields.items():
            t0 = time.perf_counter()
            f.integrate(0.01 * d["dt"], 64)
            f.sync()
            times[tuned].append(time.perf_counter() - t0)
    for f in fields.values():
        f.close()
    median = {tuned: np.median(ts) for tuned, ts in times.items()}
    assert median[True] <= 1.1 * median[False], median

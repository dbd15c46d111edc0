"""Graphs of several steps of a batch: what a new batch's first run costs, and
that runs long enough to reach them give the bits of launched steps."""
import time

import numpy as np
import pytest

from dim2d_finite_volume_b200 import workloads

pytestmark = pytest.mark.gpu
KINDS = ("periodic_xy", "hedstrom_xy", "wall_S_reflection")


@pytest.fixture(scope="module")
def F():
    from dim2d_finite_volume_b200 import field
    return field


@pytest.fixture(scope="module")
def B():
    from dim2d_finite_volume_b200 import batch
    return batch


def _fields(F, sizes):
    from dim2d_finite_volume_b200 import ic
    p = workloads.batch_params()
    out = []
    for i, n in enumerate(sizes):
        bc = KINDS[i % len(KINDS)]
        d = workloads.domain(n, n + i, T0=0.95, bubbles=[(0.0, -0.5 if "wall" in bc else 0.0, 0.15)],
                             mach=0.05 if bc == "hedstrom_xy" else 0.0, bc=bc,
                             li=ic.interface_length(0.95, p.we), we=p.we)
        f = F.Field(d["nx"], d["ny"], bc=bc, params=p)
        f.ini(d["nodes"], d["x_map"], d["y_map"])
        if "wall" in bc:
            f.apply_bc_on_nodes()
        out.append((f, d))
    return out


@pytest.mark.parametrize("steps", [8, 10, 15])
def test_first_run_of_a_new_batch(F, B, steps):
    """A run that may never be repeated does not pay for graphs that only
    repeated runs get back: at most 1.5 times the time of launched steps (twice
    that time with a capture at first use; medians of 15)."""
    fields = _fields(F, [64, 64, 64])
    times = {True: [], False: []}
    for _ in range(15):
        for graphs in times:  # in turn: the first ones load kernels and raise the clocks
            with B.Batch() as bt:
                bt.set_graphs(graphs)
                for f, d in fields:
                    bt.add(f, 0.1 * d["dt"])
                bt.sync()
                t0 = time.perf_counter()
                bt.step(steps)
                bt.sync()
                times[graphs].append(time.perf_counter() - t0)
                for f, _d in fields:
                    bt.remove(f)
    for f, _d in fields:
        f.close()
    median = {graphs: np.median(ts) for graphs, ts in times.items()}
    assert median[True] <= 1.5 * median[False], median


@pytest.mark.parametrize("schedule", [[8] * 7, [3] * 12, [1] * 13, [50, 11], [9, 9, 2, 17, 8, 8, 31]])
def test_replayed_steps_bit_identical(F, B, schedule):
    got = {}
    for graphs in (True, False):
        fields = _fields(F, [40, 33, 52, 61])
        with B.Batch() as bt:
            bt.set_graphs(graphs)
            for f, d in fields:
                bt.add(f, d["dt"])
            n0 = bt.launches
            for n in schedule:
                bt.step(n)
            bt.sync()
            got[graphs] = [f.download() for f, _d in fields] + [f.time for f, _d in fields] + \
                [bt.launches - n0]
        for f, _d in fields:
            f.close()
    for a, b in zip(got[True], got[False]):
        assert np.array_equal(a, b)

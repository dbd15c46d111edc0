"""What a stage launch does beside its strips -- wall runs, mirror and periodic
images, ghost runs and corner cells -- at the sizes where its parts meet: runs
of 28 and 29 wall columns, the corner runs of even and odd widths, strips of 30
columns, the smallest field.  Every variant of the stage kernel steps a state
that has a wall root in every column (heated wall, contact angle of 85
degrees), against the oracle.

Bars: 1e-12 normwise after one step, as in the parity tests (the wall root's
tolerance is 1e-12); after three steps 1e-11 for what its two predecessors
add.  Variants 0 to 5 evaluate every cell by the same instructions, whatever
strip, run or launch it is in, and give the same bits."""
import ctypes

import numpy as np
import pytest

from dim2d_finite_volume_b200 import workloads
from tests.test_nodebc_emulation import defined_ghost_mask

PRESETS = ["periodic_xy", "hedstrom_xy", "reflection_xy", "wall_S_reflection", "wall_S_open",
           "half_wall_S_open"]
# interior sizes: smallest field; 28/29/30/56/57/58/60 columns and one beside
SIZES = [(4, 4), (5, 4), (27, 5), (28, 16), (29, 17), (30, 31), (31, 33), (56, 9), (57, 15),
         (58, 8), (59, 7), (60, 32), (61, 33)]
WALL = dict(wall_heat_source_choice=2, wall_maximum_heat_flux=0.01, wall_heat_source_center=0.1,
            wall_heat_source_variance=0.3, wall_micro_contact_angle=85.0)


def _case(oracle, preset, n, ny):
    """(cfg, field dict, states after 1 and 3 steps) of the oracle; call with the
    wall's constants set."""
    from dim2d_finite_volume_b200 import field as F
    # with a wall: a bubble on it, an interface wide enough for a wall root on
    # the coarsest grid
    centre, li = ((0.05, -0.4), 0.5) if "wall" in preset else ((0.05, -0.1), 0.2)
    d = workloads.domain(n, ny, T0=0.95, bubbles=[centre + (0.2,)], mach=0.0, bc=preset, li=li)
    rng = np.random.default_rng(n * 100 + ny)
    q = d["nodes"]
    q[1:3] += 0.002 * rng.standard_normal(q[1:3].shape)
    if preset == "periodic_xy":
        cfg = oracle.make_cfg(d["nx"], d["ny"], periodic=True)
    else:
        ch, ty, od = F._preset(preset)
        cfg = oracle.make_cfg(d["nx"], d["ny"], bc_choice=ch, bc_type=ty, bc_order=od)
    oracle.lib().orc_clear_status()
    if preset != "hedstrom_xy":
        oracle.apply_bc_on_nodes(cfg, 0.0, d["x_map"], d["y_map"], q.copy(), q)
    states = []
    for steps in (1, 3):
        s = q.copy()
        oracle.integrate(cfg, s, d["x_map"], d["y_map"], 0.0, d["dt"], steps)
        states.append(s)
    assert oracle.lib().orc_status() == 0
    return cfg, d, states


@pytest.fixture
def wall(oracle):
    p0 = oracle.get_params()
    oracle.set_params(**WALL)
    yield WALL
    oracle.set_params(**{name: getattr(p0, name) for name, _ in p0._fields_})


def _defined(d, preset):
    """Entries of the state that the scheme defines (all but parts of the
    wall's ghost rows)."""
    m = np.ones((4, d["ny"], d["nx"]), bool)
    if "wall" in preset:
        m &= defined_ghost_mask(d["nx"], d["ny"], True) | np.pad(
            np.ones((4, d["ny"] - 4, d["nx"] - 4), bool), ((0, 0), (2, 2), (2, 2)))
    return m


@pytest.mark.parametrize("preset", PRESETS)
def test_states_have_wall_roots(oracle, wall, preset):
    """(no GPU) The cases below compare what they mean to: the oracle steps every
    one of them, and the wall's ghost density is not its first row's."""
    for n, ny in SIZES:
        _, d, states = _case(oracle, preset, n, ny)
        for s in states:
            assert np.isfinite(s[_defined(d, preset)]).all(), (n, ny)
            assert np.abs(s[_defined(d, preset)]).max() < 1e3
        if "wall" in preset:
            assert np.abs(states[1][0, 1] - states[1][0, 2]).max() > 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("preset", PRESETS)
@pytest.mark.parametrize("n,ny", SIZES)
def test_steps_match_oracle(oracle, wall, preset, n, ny):
    from dim2d_finite_volume_b200 import field as F
    cfg, d, states = _case(oracle, preset, n, ny)
    m = _defined(d, preset)
    params = F.default_params(**wall)
    bits = {}
    for variant in range(7):
        with F.Field(d["nx"], d["ny"], bc=preset, params=params) as f:
            f.ini(d["nodes"], d["x_map"], d["y_map"])
            f.variant = variant
            f.integrate(d["dt"], 1)
            got = [f.download()]
            f.integrate(d["dt"], 2)
            got.append(f.download())
        for g, ref, bar in zip(got, states, (1e-12, 1e-11)):
            for v in range(4):
                e = np.abs(g[v] - ref[v])[m[v]].max() / np.abs(ref[v][m[v]]).max()
                assert e <= bar, (variant, v, e)
        bits[variant] = got[1]
    for variant in range(1, 6):
        assert np.array_equal(bits[variant][m], bits[0][m]), variant


@pytest.mark.gpu
@pytest.mark.parametrize("preset", PRESETS)
@pytest.mark.parametrize("n,ny", [(4, 4), (5, 4), (28, 9), (29, 9), (57, 8), (59, 7), (60, 9)])
@pytest.mark.parametrize("variant", [0, 1, 5])
def test_writes_stay_in_the_field(oracle, wall, preset, n, ny, variant):
    """Guard values in the columns past the field, in both buffers that take turns
    as the state, and in the wall's ghost entries that no operator defines: as
    they were after every kind of launch."""
    import torch

    from dim2d_finite_volume_b200 import field as F
    _, d, _ = _case(oracle, preset, n, ny)
    nx, nyy = d["nx"], d["ny"]
    guard = -12345.0
    q = d["nodes"].copy()
    undefined = ~_defined(d, preset)
    q[undefined] = 77.0

    class State:
        def __init__(self, f):
            ptr, pitch = f.device_state()
            self.__cuda_array_interface__ = dict(shape=(4, nyy, pitch), typestr="<f8",
                                                 data=(ptr, False), version=3)

    with F.Field(nx, nyy, bc=preset, params=F.default_params(**wall)) as f:
        f.ini(q, d["x_map"], d["y_map"])
        f.variant = variant
        assert f.device_state()[1] > nx or nx % 16 == 0
        for _ in range(2):  # both buffers
            f.sync()
            torch.as_tensor(State(f), device="cuda")[:, :, nx:] = guard
            torch.cuda.synchronize()
            f.integrate(d["dt"], 1)
        for steps in (1, 1, 8, 3):
            f.integrate(d["dt"], steps)
            f.sync()
            s = torch.as_tensor(State(f), device="cuda").cpu().numpy()
            assert np.all(s[:, :, nx:] == guard), steps
            assert np.all(s[:, :, :nx][undefined] == 77.0), steps


@pytest.mark.gpu
@pytest.mark.parametrize("preset", ["periodic_xy", "hedstrom_xy", "wall_S_reflection",
                                    "half_wall_S_open"])
@pytest.mark.parametrize("variant", [0, 2])
def test_graphs_of_eight_steps_bit_identical(oracle, wall, preset, variant):
    """Runs long enough for every graph size, from both buffer parities."""
    from dim2d_finite_volume_b200 import field as F
    _, d, _ = _case(oracle, preset, 61, 33)
    got = []
    for graphs in (True, False):
        with F.Field(d["nx"], d["ny"], bc=preset, params=F.default_params(**wall)) as f:
            f.set_graphs(graphs)
            f.variant = variant
            f.ini(d["nodes"], d["x_map"], d["y_map"])
            n0 = f.launches
            for steps in (8, 9, 3, 16, 1, 11, 2, 8):
                f.integrate(0.5 * d["dt"], steps)
            got.append((f.download(), f.time, f.launches - n0))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


@pytest.mark.gpu
@pytest.mark.parametrize("n, ny", [(8, 8), (61, 33), (130, 64)])
@pytest.mark.parametrize("graphs", [True, False])
def test_corner_cells_in_the_launch_of_a_long_run(oracle, n, ny, graphs):
    """An untuned open field: one kernel per stage in runs of eight steps, two in
    the steps that remain and in shorter runs, with the same bits."""
    from dim2d_finite_volume_b200 import field as F
    _, d, _ = _case(oracle, "hedstrom_xy", n, ny)
    got = []
    for runs, kernels in (((16, 3), 16 * 3 + 3 * 6), ((4, 4, 4, 4, 3), 19 * 6)):
        with F.Field(d["nx"], d["ny"], bc="hedstrom_xy", params=F.default_params()) as f:
            f.set_graphs(graphs)
            f.ini(d["nodes"], d["x_map"], d["y_map"])
            n0 = f.launches
            for steps in runs:
                f.integrate(0.5 * d["dt"], steps)
            assert f.launches - n0 == kernels
            got.append((f.download(), f.compute_time_dev()))
    assert np.isfinite(got[0][0]).all()
    for v in range(2):
        assert np.array_equal(got[0][v], got[1][v])


@pytest.mark.gpu
@pytest.mark.parametrize("preset", ["periodic_xy", "hedstrom_xy", "wall_S_open"])
def test_asynchronous_copy_before_a_long_run(oracle, wall, preset):
    """A copy of the state queued before runs of eight steps and more holds that
    state, whichever buffer it is in, and the runs give what they give alone."""
    from dim2d_finite_volume_b200 import field as F
    _, d, _ = _case(oracle, preset, 60, 32)
    with F.Field(d["nx"], d["ny"], bc=preset, params=F.default_params(**wall)) as f, \
            F.Field(d["nx"], d["ny"], bc=preset, params=F.default_params(**wall)) as ref:
        for x in (f, ref):
            x.ini(d["nodes"], d["x_map"], d["y_map"])
        out = F.pinned_empty(d["nodes"].shape)
        for before, run in ((3, 8), (4, 17), (1, 9), (2, 26)):
            f.integrate(0.5 * d["dt"], before)
            f.download_async(out)
            f.integrate(0.5 * d["dt"], run)
            ref.integrate(0.5 * d["dt"], before)
            want = ref.download()
            ref.integrate(0.5 * d["dt"], run)
            f.sync()
            assert f.copy_done() and np.array_equal(out, want), (before, run)
            assert np.array_equal(f.download(), ref.download()), (before, run)


def _layer(n, ny):
    d = workloads.domain(n, ny, T0=0.95, bubbles=[(0.0, 0.0, 0.2)], mach=0.05, bc="hedstrom_xy",
                         li=0.2)
    nx, nyy = d["nx"], d["ny"]
    g = workloads.layer_map(nx, nyy, [(4, nx - 5, 4, nyy // 2), (4, nx // 2, nyy // 2, nyy - 5)])
    return d, g, (3, nx - 2), (3, nyy - 2)


@pytest.mark.gpu
@pytest.mark.parametrize("n,ny", [(60, 36), (61, 36)])
@pytest.mark.parametrize("captured", [False, True])
def test_masked_step_in_a_program_of_other_work(oracle, n, ny, captured):
    """A masked RK3 step between a program's own fills and copies, launched or
    captured into the program's graph and replayed, with NaN in the nodes that
    belong to no grid point: the oracle's result (bar 1e-11, as for a masked
    step in the masked tests)."""
    import torch

    from dim2d_finite_volume_b200 import field as F
    d, g, xb, yb = _layer(n, ny)
    nx, nyy, q = d["nx"], d["ny"], d["nodes"].copy()
    q[:, g == 0] = np.nan
    dx, dy = d["x_map"][1] - d["x_map"][0], d["y_map"][1] - d["y_map"][0]
    dt = 0.5 * d["dt"]
    ref, tmp, td = q.copy(), np.zeros_like(q), np.zeros_like(q)
    for st in (1, 2, 3):
        oracle.compute_time_dev_masked(ref, g, dx, dy, xb, yb, td)
        oracle.rk_stage_masked(st, ref, tmp, td, g, dt, xb, yb)
    src, gd = torch.from_numpy(q).cuda(), torch.from_numpy(g).cuda()
    u, tmpd, tdd = torch.empty_like(src), torch.empty_like(src), torch.empty_like(src)
    gmap = torch.empty_like(gd)
    p = F.default_params()

    def step():
        s = torch.cuda.current_stream().cuda_stream
        u.copy_(src)
        gmap.copy_(gd)
        tmpd.zero_()
        tdd.zero_()
        for st in (1, 2, 3):
            F.time_dev_masked(p, nx, nyy, u.data_ptr(), gmap.data_ptr(), dx, dy, xb, yb,
                              tdd.data_ptr(), s)
            F.rk_stage_masked(st, nx, nyy, u.data_ptr(), tmpd.data_ptr(), tdd.data_ptr(),
                              gmap.data_ptr(), dt, xb, yb, s)

    step()
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        for t in (u, tmpd, tdd):
            t.fill_(7.0)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
    got = u.cpu().numpy()
    m = g == 1
    for v in range(4):
        assert np.abs(got[v] - ref[v])[m].max() <= 1e-11 * np.abs(ref[v][m]).max(), v
    assert np.isnan(got[:, g == 0]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("preset,n", [("periodic_xy", 60), ("periodic_xy", 61),
                                      ("hedstrom_xy", 60), ("hedstrom_xy", 61)])
def test_step_noalloc_in_a_program_graph(preset, n):
    """step_noalloc captured into a program's graph, between its own copies, gives
    what the launched call gives."""
    import torch

    from dim2d_finite_volume_b200 import field as F
    d = workloads.domain(n, 44, T0=0.95, bubbles=[(0.0, 0.0, 0.2)], mach=0.0, bc=preset, li=0.2)
    L = F.library()
    L.dim2d_step_noalloc.argtypes = [ctypes.POINTER(F.Params), ctypes.c_int, ctypes.c_int,
                                     ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int),
                                     ctypes.POINTER(ctypes.c_int), ctypes.c_void_p, F._dp, F._dp,
                                     ctypes.c_double, ctypes.c_int, ctypes.c_void_p]
    arr = ctypes.c_int * 8
    ch, ty, od = F._preset(preset)
    src = torch.from_numpy(d["nodes"]).cuda()
    u = torch.empty_like(src)

    def call(steps):
        u.copy_(src)
        rc = L.dim2d_step_noalloc(ctypes.byref(F.default_params()), d["nx"], d["ny"], arr(*ch),
                                  arr(*ty), arr(*od), ctypes.c_void_p(u.data_ptr()),
                                  F._ptr(d["x_map"]), F._ptr(d["y_map"]), d["dt"], steps,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0

    for steps in (2, 3):
        call(steps)
        torch.cuda.synchronize()
        want = u.cpu().numpy()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(steps)
        u.fill_(7.0)
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(u.cpu().numpy(), want), steps

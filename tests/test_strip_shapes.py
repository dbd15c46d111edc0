"""The strip kernels at the sizes where their tiling changes: one warp's 30
columns and its neighbours' halo, the strip heights of the five shapes and
their remainders, and the 28-cell runs in which the ghost layers of open
edges are integrated -- against the oracle, over all cells that have a time
derivative (bars: 1e-12 normwise for the time derivative, as in the parity
tests; 1e-12 after two steps, whose rounding is dt times that)."""
import numpy as np
import pytest

from dim2d_finite_volume_b200 import workloads

pytestmark = pytest.mark.gpu

# interior sizes: the smallest field, one column or row short of, at and past
# a run (28), a strip (30), two of them, and a strip height (16, 32)
SIZES = [(4, 4), (27, 5), (28, 16), (29, 17), (30, 31), (31, 33), (56, 2 * 28), (57, 15), (61, 32)]


@pytest.fixture(scope="module")
def F():
    from dim2d_finite_volume_b200 import field
    return field


@pytest.mark.parametrize("preset", ["periodic_xy", "hedstrom_xy", "wall_S_open",
                                    "half_wall_S_open"])
@pytest.mark.parametrize("n,ny", SIZES)
def test_tiling_edges(oracle, F, preset, n, ny):
    d = workloads.domain(n, ny, T0=0.95, bubbles=[(0.0, -0.3, 0.2)], mach=0.05, bc=preset, li=0.2)
    rng = np.random.default_rng(n * 100 + ny)
    q = d["nodes"]
    q[1:3] += 0.02 * rng.standard_normal(q[1:3].shape)
    if preset == "periodic_xy":
        workloads.fill_periodic_ghosts(q)
        cfg = oracle.make_cfg(d["nx"], d["ny"], periodic=True)
    else:
        ch, ty, od = F._preset(preset)
        cfg = oracle.make_cfg(d["nx"], d["ny"], bc_choice=ch, bc_type=ty, bc_order=od)
        if preset != "hedstrom_xy":
            oracle.apply_bc_on_nodes(cfg, 0.0, d["x_map"], d["y_map"], q.copy(), q)
    td = oracle.compute_time_dev(cfg, 0.0, q, d["x_map"], d["y_map"])
    has = np.abs(td) < 1e30  # cells without a time derivative hold debug_real
    ref = q.copy()
    try:
        oracle.integrate(cfg, ref, d["x_map"], d["y_map"], 0.0, d["dt"], 2)
    except RuntimeError:
        # no wall root for this state, where the reference stops: its time
        # derivative is compared, no step
        assert "wall" in preset
        oracle.lib().orc_clear_status()
        ref = None
    # the wall operator leaves parts of its two ghost rows untouched
    rows = slice(2 if "wall" in preset else 0, None)
    for variant in (1, 2, 4, 5):
        with F.Field(d["nx"], d["ny"], bc=preset) as fld:
            fld.ini(q, d["x_map"], d["y_map"])
            fld.variant = variant
            got_td = fld.compute_time_dev()
            if ref is not None:
                fld.integrate(d["dt"], 2)
                got = fld.download()
        for v in range(4):
            m = has[v]
            assert np.abs(got_td[v] - td[v])[m].max() <= 1e-12 * np.abs(td[v][m]).max(), (variant, v)
            if ref is not None:
                a, b = got[v][rows], ref[v][rows]
                assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), (variant, v)


@pytest.mark.parametrize("preset", ["periodic_xy", "hedstrom_xy"])
@pytest.mark.parametrize("n,offset", [(60, 0), (60, 1), (61, 0)])
def test_caller_layouts(F, preset, n, offset):
    """dim2d_step_noalloc on the caller's array: even rows on a 16-byte boundary
    (strips), the same off it, and odd rows (tiles) give the field's own
    result (bar 1e-12, as in the no-allocation tests)."""
    import ctypes

    import torch
    d = workloads.domain(n, 44, T0=0.95, bubbles=[(0.0, 0.0, 0.2)], mach=0.05, bc=preset, li=0.2)
    with F.Field(d["nx"], d["ny"], bc=preset) as fld:
        fld.ini(d["nodes"], d["x_map"], d["y_map"])
        fld.integrate(d["dt"], 3)
        ref = fld.download()
    L = F.library()
    L.dim2d_step_noalloc.argtypes = [ctypes.POINTER(F.Params), ctypes.c_int, ctypes.c_int,
                                     ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int),
                                     ctypes.POINTER(ctypes.c_int), ctypes.c_void_p, F._dp, F._dp,
                                     ctypes.c_double, ctypes.c_int, ctypes.c_void_p]
    arr = ctypes.c_int * 8
    size = d["nodes"].size
    buf = torch.zeros(size + 2, dtype=torch.float64, device="cuda")
    dev = buf[offset:offset + size]
    dev.copy_(torch.from_numpy(d["nodes"].reshape(-1)))
    ch, ty, od = F._preset(preset)
    rc = L.dim2d_step_noalloc(ctypes.byref(F.default_params()), d["nx"], d["ny"], arr(*ch),
                              arr(*ty), arr(*od), ctypes.c_void_p(dev.data_ptr()),
                              F._ptr(d["x_map"]), F._ptr(d["y_map"]), d["dt"], 3,
                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    got = dev.cpu().numpy().reshape(d["nodes"].shape)
    for v in range(4):
        assert np.abs(got[v] - ref[v]).max() <= 1e-12 * np.abs(ref[v]).max(), v


@pytest.mark.parametrize("n,ny,offset", [(26, 9, 1), (27, 12, 0), (57, 20, 0), (61, 33, 0),
                                         (62, 33, 1)])
def test_masked_layouts(oracle, F, n, ny, offset):
    """The masked time derivative where rows cannot be copied as 16-byte pairs:
    odd nx, and even nx on an odd element, against the oracle (bar 1e-12)."""
    import torch
    d = workloads.domain(n, ny, T0=0.95, bubbles=[(0.0, 0.0, 0.2)], mach=0.05, bc="hedstrom_xy",
                         li=0.2)
    q, nx, nyy = d["nodes"], d["nx"], d["ny"]
    dx, dy = d["x_map"][1] - d["x_map"][0], d["y_map"][1] - d["y_map"][0]
    g = workloads.layer_map(nx, nyy, [(3, nx - 5, 3, nyy - 4)])
    xb, yb = (3, nx - 3), (4, nyy - 2)
    ref = np.full_like(q, 7.0)
    oracle.compute_time_dev_masked(q, g, dx, dy, xb, yb, ref)
    buf = torch.zeros(q.size + 2, dtype=torch.float64, device="cuda")
    dev = buf[offset:offset + q.size]
    dev.copy_(torch.from_numpy(q.reshape(-1)))
    gd, td = torch.from_numpy(g).cuda(), torch.full(q.shape, 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    F.time_dev_masked(F.default_params(), nx, nyy, dev.data_ptr(), gd.data_ptr(), dx, dy, xb, yb,
                      td.data_ptr())
    torch.cuda.synchronize()
    got, m = td.cpu().numpy(), g == 1
    m[:yb[0] - 1] = m[yb[1]:] = m[:, :xb[0] - 1] = m[:, xb[1]:] = False
    for v in range(4):
        assert np.abs(got[v] - ref[v])[m].max() <= 1e-12 * np.abs(ref[v][m]).max(), v
    assert np.all(got[:, ~m] == 7.0)

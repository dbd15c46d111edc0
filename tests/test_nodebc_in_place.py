"""The node pass in place (dim2d_apply_bc_on_nodes: nodes_tmp = nodes).  Its
threads are unordered, so none may read what another one writes: on the host
with every read and write recorded, and on the GPU with NaN in the ghost cells
that the pass writes."""
import os
import subprocess

import numpy as np
import pytest

from dim2d_finite_volume_b200 import workloads

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NVCC = "/usr/local/cuda/bin/nvcc"
# (south_wall, corners_y, open_w, open_e, open_n) of the node pass
FLAGS = {"wall_S_reflection": (1, 0, 0, 0, 0), "reflection_xy": (0, 1, 0, 0, 0),
         "wall_S_open": (1, 0, 1, 1, 1), "half_wall_S_open": (1, 0, 0, 1, 1)}


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("emu")
    exe = str(d / "emu")
    subprocess.check_call([NVCC, "-std=c++17", "-O1", "-w", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "include"),
                           "-o", exe, os.path.join(HERE, "emu", "emu_nodebc_in_place.cu")])
    return exe, d


def _state(preset, n, ny):
    centre, li = ((0.05, -0.4), 0.5) if "wall" in preset else ((0.05, -0.1), 0.2)
    d = workloads.domain(n, ny, T0=0.95, bubbles=[centre + (0.2,)], mach=0.0, bc=preset, li=li)
    return d


@pytest.mark.parametrize("preset", sorted(FLAGS))
@pytest.mark.parametrize("n, ny", [(4, 4), (5, 7), (40, 30)])
def test_no_thread_reads_what_another_writes(oracle, emu, preset, n, ny):
    exe, tmp = emu
    d = _state(preset, n, ny)
    p = oracle.get_params()
    got = []
    for order in (0, 1):
        fin, fout = str(tmp / "in.bin"), str(tmp / "out.bin")
        with open(fin, "wb") as fh:
            np.array([d["nx"], d["ny"], *FLAGS[preset], order], dtype=np.int32).tofile(fh)
            np.array([d["x_map"][1] - d["x_map"][0], d["y_map"][1] - d["y_map"][0], p.re, p.we,
                      p.pr, p.cv_r, np.cos(np.deg2rad(p.wall_micro_contact_angle)),
                      d["x_map"][0]]).tofile(fh)
            d["nodes"].tofile(fh)
        out = subprocess.check_output([exe, fin, fout]).decode()
        stats = dict(kv.split("=") for kv in out.split())
        assert stats["bad"] == "0" and stats["race"] == "0", out
        got.append(np.fromfile(fout))
    assert np.array_equal(got[0], got[1], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("preset", ["wall_S_reflection", "half_wall_S_open", "reflection_xy"])
@pytest.mark.parametrize("n, ny", [(4, 4), (61, 33), (213, 213)])
def test_mirror_ghosts_that_are_not_numbers(preset, n, ny):
    """What a mirror side's ghost cells held before the pass does not matter."""
    from dim2d_finite_volume_b200 import field as F
    d = _state(preset, n, ny)
    got = []
    for ghosts in (None, np.nan):
        q = d["nodes"].copy()
        if ghosts is not None:
            q[:, 2:-2, :2] = ghosts
            if preset != "half_wall_S_open":
                q[:, 2:-2, -2:] = ghosts
        with F.Field(d["nx"], d["ny"], bc=preset) as f:
            f.ini(q, d["x_map"], d["y_map"])
            f.apply_bc_on_nodes()
            got.append(f.download())
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1])

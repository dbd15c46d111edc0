"""The south wall's momentum flux in mixed precision: FP64 from the face's sums
on.  A state of rest, uniform, whose density and pressure are FP32 numbers, so
that the FP32 face pass of the rows above is exact: what a heated wall gives
the first row is then the oracle's value to FP64 rounding (some 1e-16 of
P / dy; bar 1e-13, where a flux rounded to FP32 is up to 6e-8 off)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
R, P = 0.5, 0.2890625  # density and pressure


@pytest.fixture(scope="module")
def F():
    from dim2d_finite_volume_b200 import field
    return field


@pytest.mark.parametrize("preset", ["wall_S_reflection", "wall_S_open", "half_wall_S_open"])
@pytest.mark.parametrize("heat", [0.013, -0.0071])
def test_heated_wall_flux(oracle, F, preset, heat):
    from dim2d_finite_volume_b200 import ic
    nx, ny, x_map, y_map = ic.grid(35, 21)
    params = F.default_params(wall_heat_source_choice=1, wall_maximum_heat_flux=heat)
    q = np.zeros((4, ny, nx))
    q[0] = R
    # P = 3/cv_r W/(3 - rho) - 3 rho^2 with W = E + 3 rho^2 at rest
    q[3] = (P + 3.0 * R * R) * (3.0 - R) * params.cv_r / 3.0 - 3.0 * R * R
    ch, ty, od = F._preset(preset)
    cfg = oracle.make_cfg(nx, ny, bc_choice=ch, bc_type=ty, bc_order=od)
    p0 = oracle.get_params()
    oracle.set_params(wall_heat_source_choice=1, wall_maximum_heat_flux=heat)
    try:
        ref = oracle.compute_time_dev(cfg, 0.0, q, x_map, y_map)
    finally:
        oracle.set_params(**{name: getattr(p0, name) for name, _ in p0._fields_})
    inner = (slice(None), slice(2, -2), slice(2, -2))
    scale = P / (y_map[1] - y_map[0])
    assert np.abs(ref[2, 2, 2:-2]).min() > 1e-3 * scale  # the heat moves the first row
    for variant in range(6):
        with F.Field(nx, ny, bc=preset, params=params, precision=F.MIXED) as fld:
            fld.ini(q, x_map, y_map)
            fld.variant = variant
            got = fld.compute_time_dev()
        assert np.abs(got - ref)[inner][2].max() <= 1e-13 * scale, variant

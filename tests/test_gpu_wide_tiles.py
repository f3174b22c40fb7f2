"""Tiles with several warps side by side (they share two columns) against the general path, a
separate kernel chain that evaluates every cell on its own: grids whose last column falls on
a shared column, on the ones next to it, and one strip's width apart."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from helpers import grid_coords, random_re_case  # noqa: E402

PLANES = ("h", "hu", "hv", "z_b", "G")


def sides(ny, nx):
    """An inflow and a bed handler on the east side: its ring cells keep the depth of their own
    update.  The reflective sides end one cell short of it, so its corners are nodata."""
    def side(t, x0, x1, y0, y1, normal, values=(0.0, 0.0, 0.0, 0.0)):
        poly = [[x0 - 0.5, y0 - 0.5], [x1 + 0.5, y0 - 0.5], [x1 + 0.5, y1 + 0.5], [x0 - 0.5, y1 + 0.5]]
        return {"type": t, "polygon": poly, "values": list(values), "normal": list(normal)}

    return {
        "east": side("ConstantInflux", nx - 1, nx - 1, 1, ny - 2, [1.0, 0.0], (0.3, -1.0, 0.0, 0.0)),
        "east_bed": side("TransmissiveBed", nx - 1, nx - 1, 1, ny - 2, [1.0, 0.0]),
        "west": side("Transmissive", 0, 0, 0, ny - 1, [-1.0, 0.0]),
        "south": side("Reflective", 0, nx - 2, 0, 0, [0.0, -1.0]),
        "north": side("Reflective", 0, nx - 2, ny - 1, ny - 1, [0.0, 1.0]),
    }


def case(ny, nx, regime, mpm):
    arrs, params, X, Y, _ = random_re_case(ny, nx, seed=ny + 3 * nx, regime=regime, mpm=mpm)
    if regime == "wetdry":  # a dry last column above the water in front of it, every other row
        arrs["h"][::2, nx - 1] = 0.0
        arrs["z"][::2, nx - 1] += 0.6
    return arrs, dict(params, boundaries=sides(ny, nx)), X, Y


def run(arrs, params, X, Y, dtype, path, rows, warps, steps):
    from pyexner_b200 import BoundaryManager, RoeExnerState, _lib, create_solver_bundle, run_steps
    from pyexner_b200.cases import seds_matrix
    from pyexner_b200.solvers import _re_plan

    bounds = BoundaryManager(params, X, Y)
    st = RoeExnerState.from_numpy(arrs, seds_matrix(params["erosion"]), dtype=dtype)
    bundle = create_solver_bundle("Roe Exner")
    cfg = bundle.config(st, None, bounds, 0.1, dict(params, stage_path=path, band_rows=rows))
    mask = bundle.mask_fn(st, None, bounds.boundary_mask)
    st = bundle.init_fn(st, mask, cfg)
    assert _lib.load().pxb_re_plan_tile_warps(_re_plan(st, mask, cfg).handle) == warps
    dts = run_steps(st, mask, cfg, "SSPRK2", steps, 0.5).cpu().numpy()
    return dts, st.to_numpy()


# warps side by side w, index of the last column in the last tile: 30, 60 and 90 are the columns
# that two warps share, the second of them without their west face; (ny, nx, band_rows) is a
# small grid for which the cheapest tiling has that shape on 148 SMs
F64 = {(2, 29): (120, 478, 2), (2, 30): (120, 479, 2), (2, 31): (120, 480, 2), (2, 60): (260, 117, 2),
       (2, 61): (60, 510, 2), (4, 30): (120, 263, 2), (4, 31): (120, 264, 2), (4, 60): (100, 293, 2),
       (4, 61): (100, 294, 2), (4, 89): (100, 322, 2), (4, 90): (100, 323, 2), (4, 91): (100, 324, 2)}
F32 = {(2, 29): (80, 590, 2), (2, 30): (40, 1151, 2), (2, 31): (40, 1152, 2), (3, 60): (140, 1351, 8),
       (3, 61): (140, 1352, 8), (3, 89): (260, 176, 2), (3, 90): (260, 177, 2), (3, 91): (260, 178, 2),
       (4, 30): (100, 495, 2), (4, 60): (160, 293, 2), (4, 90): (40, 1251, 2)}


@pytest.mark.parametrize("regime,mpm", [("fast", True), ("wetdry", False)])
@pytest.mark.parametrize("warps,last", sorted(F64))
def test_float64_gives_the_general_path_bits(warps, last, regime, mpm):
    ny, nx, rows = F64[warps, last]
    assert (nx - 1 - last) % (30 * warps - 4) == 0
    arrs, params, X, Y = case(ny, nx, regime, mpm)
    a = run(arrs, params, X, Y, "float64", "fused", rows, warps, 3)
    b = run(arrs, params, X, Y, "float64", "general", 0, 0, 3)
    assert np.array_equal(a[0], b[0], equal_nan=True)
    for f in PLANES:
        assert np.array_equal(a[1][f], b[1][f], equal_nan=True), f


@pytest.mark.parametrize("warps,last", sorted(F32))
def test_float32_stays_at_the_general_path(warps, last):
    """Two steps, a few roundings of each apart: 1e-6 normwise, as the other tilings are held to."""
    ny, nx, rows = F32[warps, last]
    assert (nx - 1 - last) % (30 * warps - 4) == 0
    arrs, params, X, Y = case(ny, nx, "smooth", True)
    a = run(arrs, params, X, Y, "float32", "fused", rows, warps, 2)
    b = run(arrs, params, X, Y, "float32", "general", 0, 0, 2)
    for f in PLANES:
        x, y = a[1][f], b[1][f]
        assert np.max(np.abs(x - y)) <= 1e-6 * max(1e-3, np.max(np.abs(y))), f


@pytest.mark.parametrize("rows", [500, 2**31 - 1])
def test_bands_taller_than_the_grid(rows):
    """band_rows beyond the grid's rows asks for bands as tall as they get: the same bits."""
    arrs, params, X, Y = case(80, 70, "fast", True)
    a = run(arrs, params, X, Y, "float64", "fused", rows, 1, 2)
    b = run(arrs, params, X, Y, "float64", "general", 0, 0, 2)
    for f in PLANES:
        assert np.array_equal(a[1][f], b[1][f], equal_nan=True), f

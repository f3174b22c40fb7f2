"""Tile edges of the fused stage kernel: grids whose last strip, last band or share of rows
per warp is as short or as long as it gets, against the general path (a separate kernel
chain that evaluates every cell on its own) and over band heights."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from helpers import random_re_case  # noqa: E402

PLANES = ("h", "hu", "hv", "z_b", "G")


def run(arrs, params, X, Y, dtype, path, rows, steps=3, scheme="SSPRK2"):
    from pyexner_b200 import BoundaryManager, RoeExnerState, create_solver_bundle, run_steps
    from pyexner_b200.cases import seds_matrix

    bounds = BoundaryManager(params, X, Y)
    st = RoeExnerState.from_numpy(arrs, seds_matrix(params["erosion"]), dtype=dtype)
    bundle = create_solver_bundle("Roe Exner")
    cfg = bundle.config(st, None, bounds, 0.1, dict(params, stage_path=path, band_rows=rows))
    mask = bundle.mask_fn(st, None, bounds.boundary_mask)
    st = bundle.init_fn(st, mask, cfg)
    dts = run_steps(st, mask, cfg, scheme, steps, 0.5).cpu().numpy()
    return dts, st.to_numpy()


# strips of wx warps own 30 wx - 4 columns, the first 3 more and the last up to 3 more:
# 32 / 33, 58 / 59, 62 / 63, 122 / 123 columns are one strip and the first two-strip grid for
# wx = 1, 1 (two strips), 2 and 4; bands of 2 rows are the shortest, rows = 3 leaves short
# and long ones, and warps whose share of a band is empty
@pytest.mark.parametrize("ny,nx,rows", [(9, 32, 2), (10, 33, 3), (37, 58, 0), (5, 59, 2), (64, 62, 7), (21, 63, 64),
                                        (17, 122, 5), (130, 123, 0), (300, 7, 0), (4, 400, 2)])
@pytest.mark.parametrize("bc,regime,mpm", [("trans_x_refl_y", "fast", True), ("influx_left", "wetdry", False),
                                           ("partial_nodata", "wetdry", True), ("refl_self", "smooth", True)])
def test_tile_edges_give_the_general_path_bits(ny, nx, rows, bc, regime, mpm):
    """float64: the fused path's dts and planes equal the general path's bit for bit."""
    arrs, params, X, Y, _ = random_re_case(ny, nx, seed=ny + 3 * nx, regime=regime, bcname=bc, mpm=mpm)
    a = run(arrs, params, X, Y, "float64", "fused", rows)
    b = run(arrs, params, X, Y, "float64", "general", 0)
    assert np.array_equal(a[0], b[0], equal_nan=True)
    for f in PLANES:
        assert np.array_equal(a[1][f], b[1][f], equal_nan=True), f


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("ny,nx", [(70, 33), (141, 260)])
def test_no_handlers_at_all(ny, nx, dtype):
    """A plan without boundary handlers: the ring is nodata and the fused path reads nothing
    beyond the grid.  One Forward-Euler and two averaged steps against the general path
    (float64: the same bits; float32: a few roundings of each step, 1e-6 normwise)."""
    arrs, params, X, Y, _ = random_re_case(ny, nx, seed=5, regime="smooth")
    params["boundaries"] = {}
    for scheme, steps in (("FE", 1), ("SSPRK2", 2)):
        a = run(arrs, params, X, Y, dtype, "fused", 0, steps, scheme)
        b = run(arrs, params, X, Y, dtype, "general", 0, steps, scheme)
        for f in PLANES:
            x, y = a[1][f], b[1][f]
            if dtype == "float64":
                assert np.array_equal(x, y, equal_nan=True), f
            else:
                assert np.max(np.abs(x - y)) <= 1e-6 * max(1e-3, np.max(np.abs(y))), f

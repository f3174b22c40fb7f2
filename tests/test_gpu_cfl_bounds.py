"""Wide CFL items (bounds per row, exact speeds only where a row may hold the maximum)
against the narrow ones (every face): the same dt bit for bit on fields where the bounds
are tight, loose, tied, or where only a single face decides."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bc_specs import BC_SPECS, grid_coords  # noqa: E402


def fields(kind, ny, nx, rng):
    h = rng.uniform(0.2, 0.5, (ny, nx))
    u, v = rng.uniform(-0.5, 0.5, (2, ny, nx))
    if kind == "uniform":  # every face ties
        h[:], u[:], v[:] = 0.3, 0.7, 0.0
    elif kind == "rest":
        u[:] = v[:] = 0.0
    elif kind == "supercritical":  # one real root in places: the clipped cubic
        u += 4.0
    elif kind == "drops":  # dry cells among fast thin ones
        h[rng.random((ny, nx)) < 0.3] = 0.0
        h[rng.random((ny, nx)) < 0.1] = 2e-4
        u *= 3.0
    elif kind == "peak":  # a single deep cell in the last row and column but one
        h *= 0.1
        h[ny - 2, nx - 2] = 2.0
    elif kind == "nan":
        h[ny // 2, nx // 3] = np.nan
    return h, h * u, h * v


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("g", [0.0, 0.005, 0.5])
@pytest.mark.parametrize("kind", ["uniform", "rest", "supercritical", "drops", "peak", "nan", "plain"])
def test_wide_items_give_the_narrow_items_dt(kind, g, dtype):
    """The allocation-free entry point takes narrow items at every size; the plan takes wide
    ones here (1.3 M cells; strips of 124 columns with a short last one)."""
    import ctypes

    from pyexner_b200 import BoundaryManager, RoeExnerState, _lib, create_solver_bundle

    ny, nx = 1070, 1217
    rng = np.random.default_rng(7)
    h, hu, hv = fields(kind, ny, nx, rng)
    G = g * rng.uniform(0.5, 1.0, h.shape)
    zero = np.zeros_like(h)
    params = dict(flux_scheme="Roe Exner", boundaries=BC_SPECS["trans_x_refl_y"](ny, nx), erosion=dict(grass_factor=0.005))
    X, Y = grid_coords(ny, nx)
    st = RoeExnerState.from_numpy(dict(h=h, hu=hu, hv=hv, z=zero, z_b=zero + 0.1, n=zero, G=G), np.zeros((1, 1)), dtype)
    bundle = create_solver_bundle("Roe Exner")
    cfg = bundle.config(st, None, BoundaryManager(params, X, Y), 0.1, params)
    mask = bundle.mask_fn(st, None, cfg.boundaries.boundary_mask)
    wide = bundle.compute_dt_fn(st, 0.5, mask, cfg)
    narrow = torch.empty((), dtype=dtype, device="cuda")
    _lib.call("pxb_re_cfl_noalloc", ny, nx, st.pitch, _lib.F32 if dtype == torch.float32 else _lib.F64, 0.1, 0.5,
              st.h.data_ptr(), st.hu.data_ptr(), st.hv.data_ptr(), st.G.data_ptr(), None, narrow.data_ptr(),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    a, b = wide.cpu().numpy(), narrow.cpu().numpy()
    assert a.tobytes() == b.tobytes() or (np.isnan(a) and np.isnan(b)), (a, b)

"""States whose planes are column windows of wider tensors: row pitches other than the
wrapper's own, and planes that end with their last cell."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bc_specs import BC_SPECS, grid_coords  # noqa: E402

FIELDS = ("h", "hu", "hv", "z", "z_b", "n", "n_b", "G")
X0 = 32  # first column of the windows: 16-byte aligned rows


def setup(ny, nx, dtype, width):
    """A channel state, its copy in windows of (ny, width) tensors, and what drives them."""
    from pyexner_b200 import BoundaryManager, RoeExnerState, create_solver_bundle

    rng = np.random.default_rng(ny + nx)
    h = rng.uniform(0.2, 0.5, (ny, nx))
    u, v = rng.uniform(-0.5, 0.5, (2, ny, nx))
    arrs = dict(h=h, hu=h * u, hv=h * v, z=np.zeros_like(h), z_b=np.full_like(h, 0.1), G=0.005 * rng.uniform(0.5, 1, h.shape))
    params = dict(flux_scheme="Roe Exner", boundaries=BC_SPECS["trans_x_refl_y"](ny, nx), erosion=dict(grass_factor=0.005))
    X, Y = grid_coords(ny, nx)
    st = RoeExnerState.from_numpy(arrs, np.zeros((1, 1)), dtype)
    bundle = create_solver_bundle("Roe Exner")
    cfg = bundle.config(st, None, BoundaryManager(params, X, Y), 0.1, params)
    mask = bundle.mask_fn(st, None, cfg.boundaries.boundary_mask)
    st = bundle.init_fn(st, mask, cfg)
    whole = {f: torch.full((ny, width), 7.0, dtype=dtype, device="cuda") for f in FIELDS}
    win = st.replace(**{f: whole[f][:, X0:X0 + nx] for f in FIELDS})
    for f in FIELDS:
        getattr(win, f).copy_(getattr(st, f))
    return bundle, cfg, mask, st, win, whole


# the windows end at the last column of their tensors, or one column before it: the last group
# of four columns is whole or partial
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("nx,width", [(1220, 1252), (1219, 1252), (1217, 1249)])
def test_dt_of_a_window(nx, width, dtype):
    """Above the size where the CFL takes wide items (the third pitch allows no 16-byte loads)."""
    bundle, cfg, mask, st, win, _ = setup(1070, nx, dtype, width)
    assert win.h.stride(0) == width and win.h.storage_offset() == X0
    assert torch.equal(bundle.compute_dt_fn(win, 0.5, mask, cfg), bundle.compute_dt_fn(st, 0.5, mask, cfg))

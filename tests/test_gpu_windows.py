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


def same(a, b, fields=("h", "hu", "hv", "z_b", "G")):
    for f in fields:
        assert torch.equal(getattr(a, f), getattr(b, f)), f


def outside_untouched(whole, nx):
    for f, t in whole.items():
        assert bool((t[:, :X0] == 7.0).all()) and bool((t[:, X0 + nx:] == 7.0).all()), f


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("path", ["fused", "general"])
def test_stage_and_steps_of_a_window(path, dtype):
    """What the wrapper allocates for a window has the window's pitch: the same bits as the
    state's own, and nothing outside the window changes."""
    from pyexner_b200 import run_steps

    nx, width = 70, 200  # (70 columns alone would be padded to 96)
    bundle, cfg, mask, st, win, whole = setup(41, nx, dtype, width)
    cfg = cfg._replace(stage_path={"fused": 1, "general": 2}[path], plans={})
    dt = float(bundle.compute_dt_fn(st, 0.5, mask, cfg))
    same(bundle.step_fn(win, 0.0, dt, mask, cfg), bundle.step_fn(st, 0.0, dt, mask, cfg))
    assert torch.equal(run_steps(win, mask, cfg, "FE", 3, 0.5), run_steps(st, mask, cfg, "FE", 3, 0.5))
    same(win, st)
    outside_untouched(whole, nx)


def test_plain_roe_step_of_a_window():
    from pyexner_b200 import RoeState

    from bc_specs import ROE_BC_SPECS
    from pyexner_b200 import BoundaryManager, create_solver_bundle

    ny, nx, width = 41, 70, 200
    rng = np.random.default_rng(1)
    h = rng.uniform(0.3, 0.6, (ny, nx))
    X, Y = grid_coords(ny, nx)
    params = dict(flux_scheme="Roe", boundaries=ROE_BC_SPECS[sorted(ROE_BC_SPECS)[0]](ny, nx))
    st = RoeState.from_numpy(dict(h=h, hu=0.2 * h, hv=-0.1 * h, z=0.0 * h, n=0.01 + 0.0 * h), torch.float64)
    whole = {f: torch.full((ny, width), 7.0, dtype=torch.float64, device="cuda") for f in RoeState.PLANES}
    win = st.replace(**{f: whole[f][:, X0:X0 + nx].copy_(getattr(st, f)) for f in RoeState.PLANES})
    bundle = create_solver_bundle("Roe")
    cfg = bundle.config(st, None, BoundaryManager(params, X, Y), 0.1, params)
    mask = bundle.mask_fn(st)
    dt = float(bundle.compute_dt_fn(st, 0.5, mask, cfg))
    assert float(bundle.compute_dt_fn(win, 0.5, mask, cfg)) == dt
    same(bundle.step_fn(win, 0.0, dt, mask, cfg), bundle.step_fn(st, 0.0, dt, mask, cfg), RoeState.PLANES)
    outside_untouched(whole, nx)


def test_reverse_mode_of_a_window():
    """The adjoint comes back in the window's columns alone.  Its atomic sums vary in their last
    bits: 1e-12 normwise."""
    from pyexner_b200.tangent import vjp_run

    nx, width = 70, 200
    _, cfg, mask, st, win, whole = setup(41, nx, torch.float64, width)
    gen = torch.Generator(device="cuda").manual_seed(3)
    abar = st.clone()
    for f in FIELDS:
        getattr(abar, f).copy_(torch.randn(st.shape, generator=gen, dtype=torch.float64, device="cuda"))
    bars = {f: torch.full((41, width), 7.0, dtype=torch.float64, device="cuda") for f in FIELDS}
    wbar = abar.replace(**{f: bars[f][:, X0:X0 + nx].copy_(getattr(abar, f)) for f in FIELDS})
    vjp_run(st, abar, mask, cfg, 3, "SSPRK2", 0.5, checkpoint_every=2)
    vjp_run(win, wbar, mask, cfg, 3, "SSPRK2", 0.5, checkpoint_every=2)
    for f in ("h", "hu", "hv", "z_b", "G"):
        a, b = getattr(abar, f), getattr(wbar, f)
        assert float((a - b).abs().max()) <= 1e-12 * float(a.abs().max()), f
    outside_untouched(whole, nx)
    outside_untouched(bars, nx)

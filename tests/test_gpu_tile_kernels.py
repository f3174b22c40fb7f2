"""Edges of the tiled kernels (16 x 8 cells a block: plain Roe stage, general path's faces,
reverse mode) and of the one-launch boundary handlers, against the oracle or, for the
reverse mode, the transpose identity with the tangent model."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from helpers import ROE_BC_SPECS, grid_coords, oracle_setup, random_re_case, rel_err  # noqa: E402
from oracle import boundaries as OB  # noqa: E402
from oracle import integrators as OI  # noqa: E402
from oracle import roe_exner as ORE  # noqa: E402

# one tile, one cell over, just under and at two tiles, a tile of the fewest cells
EDGES = [(8, 16), (9, 17), (15, 31), (16, 33), (5, 100), (65, 6)]


@pytest.mark.parametrize("ny,nx", EDGES)
@pytest.mark.parametrize("bc", sorted(ROE_BC_SPECS))
def test_plain_roe_tiles(ny, nx, bc):
    """Four float64 SSPRK2 steps: 1e-10 normwise, the bound of the golden Roe runs."""
    from pyexner_b200 import BoundaryManager, RoeState, create_solver_bundle, run_steps

    rng = np.random.default_rng(ny * 101 + nx)
    h = rng.uniform(0.3, 0.6, (ny, nx))
    arrs = dict(h=h, hu=h * rng.uniform(-0.5, 0.5, (ny, nx)), hv=h * rng.uniform(-0.5, 0.5, (ny, nx)),
                z=rng.uniform(0.0, 0.05, (ny, nx)), n=rng.uniform(0.0, 0.03, (ny, nx)))
    X, Y = grid_coords(ny, nx)
    spec = ROE_BC_SPECS[bc](ny, nx)
    params = dict(flux_scheme="Roe", boundaries=spec)
    bm = BoundaryManager(params, X, Y)
    st = RoeState.from_numpy(arrs, torch.float64)
    bundle = create_solver_bundle("Roe")
    cfg = bundle.config(st, None, bm, 0.1, params)
    mask = bundle.mask_fn(st)
    st = bundle.init_fn(st, mask, cfg)
    dts = run_steps(st, mask, cfg, "SSPRK2", 4, 0.5)
    ost, odts = OI.run_roe({k: np.array(v) for k, v in arrs.items()}, OB.Boundaries("Roe", spec, X, Y), 0.1, 0.5, 4,
                           "SSPRK2")
    assert rel_err(dts.cpu().numpy(), odts) <= 1e-10
    got = st.to_numpy()
    for f in ("h", "hu", "hv", "z", "n"):
        assert rel_err(got[f], ost[f]) <= 1e-10, f


@pytest.mark.parametrize("ny,nx", EDGES)
def test_reverse_mode_tiles(ny, nx):
    """<abar_0, du_0> == <abar_N, J du_0> over 3 steps (1e-9, as on the larger grids)."""
    from pyexner_b200.tangent import jvp_run, vjp_run
    from test_gpu_tangent import inner, random_adjoint, setup, smooth_case, tangent_state

    _, cfg, mask, st = setup(*smooth_case(ny, nx))
    rng = np.random.default_rng(3)
    du = tangent_state(st, rng, ("h", "hu", "hv", "z_b"))
    s, td = st.clone(), du.clone()
    jvp_run(s, td, mask, cfg, 3, "SSPRK2", 0.5)
    abar = random_adjoint(st, rng)
    rhs = inner(abar, td)
    a0 = vjp_run(st, abar.clone(), mask, cfg, 3, "SSPRK2", 0.5, checkpoint_every=2)
    lhs = inner(a0, du, ("h", "hu", "hv", "z_b"))
    assert abs(lhs - rhs) <= 1e-9 * max(abs(rhs), 1e-30)


def walls(ny, nx, parts):
    """Each side in `parts` pieces that overlap by a cell or more, so that some cells are
    written by several handlers and some are the donors of a later one; two handlers with
    disjoint fields on the first piece of each side."""
    def cuts(n):
        e = np.linspace(0, n, parts + 1).astype(int)
        return [(max(0, e[k] - 1) - 0.5, e[k + 1] - 0.5) for k in range(parts)]

    out = {}
    for side, normal, n in (("west", [-1.0, 0.0], ny), ("east", [1.0, 0.0], ny), ("south", [0.0, -1.0], nx),
                            ("north", [0.0, 1.0], nx)):
        for k, (p0, p1) in enumerate(cuts(n)):
            x0, x1, y0, y1 = {"west": (-0.5, 0.5, p0, p1), "east": (nx - 1.5, nx - 0.5, p0, p1),
                              "south": (p0, p1, -0.5, 0.5), "north": (p0, p1, ny - 1.5, ny - 0.5)}[side]
            poly = [[x0, y0], [x1, y0], [x1, y1], [x0, y1]]
            for t in (("Transmissive", "TransmissiveBed") if k == 0 else ("Reflective",)):
                out[f"{side}{k}{t}"] = dict(type=t, polygon=poly, values=[0.0] * 4, normal=normal)
    return out


# 8 and 24 handlers (one launch, and more than the 16 of a launch), a level of one block and
# of 8 blocks' cells, a level above the cluster's 4096 cells (a launch per handler)
@pytest.mark.parametrize("ny,nx,parts", [(9, 11, 1), (40, 33, 5), (300, 420, 3), (800, 1100, 2), (900, 1200, 1)])
@pytest.mark.parametrize("dtype,tol", [("float64", 1e-12), ("float32", 2e-5)])
def test_handlers_of_a_layout(ny, nx, parts, dtype, tol):
    """One stage of the general path after the init, against the oracle's handlers one after
    the other (the bounds of the general path's other stages)."""
    from pyexner_b200 import BoundaryManager, RoeExnerState, create_solver_bundle
    from pyexner_b200.boundaries import index_coords
    from pyexner_b200.cases import seds_matrix

    arrs, params, _, _, mpm = random_re_case(ny, nx, seed=ny + nx, regime="smooth", mpm=False)
    X, Y = index_coords(ny, nx)
    params = dict(params, boundaries=walls(ny, nx, parts), stage_path="general")
    seds = seds_matrix(params["erosion"])
    ost, omask, obcs = oracle_setup(arrs, params, X, Y, mpm, seds)
    odt = ORE.compute_dt(ost, 0.5, 0.1, omask[0])
    o1 = ORE.stage(ost, odt, 0.1, omask, obcs, mpm, 0.0)
    bm = BoundaryManager(params, X, Y)
    st = RoeExnerState.from_numpy(arrs, seds, dtype=dtype)
    bundle = create_solver_bundle("Roe Exner")
    cfg = bundle.config(st, None, bm, 0.1, params)
    mask = bundle.mask_fn(st, None, bm.boundary_mask)
    st = bundle.init_fn(st, mask, cfg)
    got = bundle.step_fn(st, 0.0, float(odt), mask, cfg).to_numpy()
    for f in ("h", "hu", "hv", "z_b", "n", "G"):
        assert rel_err(got[f], o1[f]) <= tol, f

"""The allocation-free CFL entry point above the size where it takes wide items: the plan's dt
bit for bit, call after call, with calls on small grids (the other kernel, the same scratch
array) in between, and no device memory allocated."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bc_specs import BC_SPECS, grid_coords  # noqa: E402


def case(ny, nx, dtype, layout, g):
    from pyexner_b200 import BoundaryManager, RoeExnerState, create_solver_bundle
    from pyexner_b200.state import alloc_plane

    rng = np.random.default_rng(ny)
    h = rng.uniform(0.2, 0.5, (ny, nx))
    h[rng.random((ny, nx)) < 0.05] = 0.0
    u, v = rng.uniform(-0.5, 0.5, (2, ny, nx))
    arrs = dict(h=h, hu=h * u, hv=h * v, z=np.zeros_like(h), z_b=np.full_like(h, 0.1), G=g * rng.uniform(0.5, 1, h.shape))
    params = dict(flux_scheme="Roe Exner", boundaries=BC_SPECS[layout](ny, nx), erosion=dict(grass_factor=g))
    X, Y = grid_coords(ny, nx)
    st = RoeExnerState.from_numpy(arrs, np.zeros((1, 1)), dtype)
    bundle = create_solver_bundle("Roe Exner")
    cfg = bundle.config(st, None, BoundaryManager(params, X, Y), 0.1, params)
    mask = bundle.mask_fn(st, None, cfg.boundaries.boundary_mask)
    nodata = None
    if bool(mask[0].any()):
        nodata = alloc_plane(ny, nx, torch.uint8, "cuda", align=st.pitch)
        nodata.copy_(mask[0].to(torch.uint8))
    return st, nodata, bundle.compute_dt_fn(st, 0.5, mask, cfg)


# 4.02 M cells with a short last strip and band; 3.99 M cells, just below the line
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("layout,g", [("trans_x_refl_y", 0.0), ("partial_nodata", 0.005)])
def test_large_grids(layout, g, dtype):
    from pyexner_b200 import _lib

    cases = [case(ny, nx, dtype, layout, g) for ny, nx in ((2003, 2007), (1993, 2003), (60, 70))]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = torch.empty((), dtype=dtype, device="cuda")
    for turn in range(2):
        for st, nodata, ref in cases:
            out.fill_(-1.0)
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            ny, nx = st.shape
            _lib.call("pxb_re_cfl_noalloc", ny, nx, st.pitch, _lib.F32 if dtype == torch.float32 else _lib.F64, 0.1, 0.5,
                      st.h.data_ptr(), st.hu.data_ptr(), st.hv.data_ptr(), st.G.data_ptr(),
                      nodata.data_ptr() if nodata is not None else None, out.data_ptr(), stream)
            torch.cuda.synchronize()
            assert torch.equal(out, ref), (turn, ny, nx)
            if turn:
                assert torch.cuda.mem_get_info()[0] == free

"""Reverse mode at the edges of its inputs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_tangent import random_adjoint, setup, smooth_case  # noqa: E402


def test_parameter_adjoints_with_a_fraction_of_zero():
    """No sediment in the class: G is 0 whatever the other constants are, so the gradients of the
    grain diameter, density, threshold and porosity are 0 (that of the fraction itself is not
    defined: n_p_mix is the sixth root of the mean of d50 times the fraction)."""
    from pyexner_b200.tangent import ParamAdjoints, vjp_run

    arrs, params, X, Y = smooth_case()
    params["erosion"]["sediments"]["s1"]["fraction"] = 0.0
    _, cfg, mask, st = setup(arrs, params, X, Y)
    pa = ParamAdjoints(cfg, st.seds)
    abar = vjp_run(st, random_adjoint(st, np.random.default_rng(2)), mask, cfg, 4, "SSPRK2", 0.5, params=pa)
    assert np.all(pa.seds_bar[1:] == 0.0), pa.seds_bar
    for f in ("h", "hu", "hv", "z_b"):
        assert bool(torch.isfinite(getattr(abar, f)).all()), f


def test_no_memory_is_kept_after_a_run():
    """What a run needs goes back to torch's allocator: the plan holds nothing between calls."""
    from pyexner_b200.tangent import vjp_run

    def go(ny, nx, every):
        _, cfg, mask, st = setup(*smooth_case(ny, nx))
        abar = random_adjoint(st, np.random.default_rng(4))
        free = []
        for k in range(2):  # (the first call loads kernels)
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            free.append(torch.cuda.mem_get_info()[0])
            vjp_run(st, abar, mask, cfg, 4, "SSPRK2", 0.5, checkpoint_every=every)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return free + [torch.cuda.mem_get_info()[0]]

    go(26, 34, 4)
    free = go(400, 400, 4)  # a workspace of about 90 MB
    assert free[0] - free[2] < 32 << 20, free


def test_workspace_of_the_c_call():
    """The run in a caller's workspace against the run that allocates its own (the adjoint's
    atomic sums vary in their last bits: 1e-12 normwise), and what is refused."""
    import ctypes

    from pyexner_b200 import _lib
    from pyexner_b200.solvers import _re_plan, _stream

    _, cfg, mask, st = setup(*smooth_case(40, 50))
    plan = _re_plan(st, mask, cfg)
    size = ctypes.c_size_t()
    _lib.call("pxb_re_vjp_workspace_size", plan.handle, 5, 2, ctypes.byref(size))
    work = torch.empty(size.value + 256, dtype=torch.uint8, device="cuda")
    a = random_adjoint(st, np.random.default_rng(4))
    b = a.clone()

    def args(bar):
        return (plan.handle, ctypes.byref(st.c_fields()), 5, _lib.SSPRK2, 0.5, 0.0, 2, ctypes.byref(bar.c_fields()))

    _lib.call("pxb_re_vjp_run", *args(a), _stream())
    for ptr, n in ((work.data_ptr(), size.value - 1), (work.data_ptr() + 8, size.value)):
        with pytest.raises(_lib.PxbError):
            _lib.call("pxb_re_vjp_run_in", *args(b), None, ctypes.c_void_p(ptr), n, _stream())
    _lib.call("pxb_re_vjp_run_in", *args(b), None, ctypes.c_void_p(work.data_ptr()), size.value, _stream())
    for f in ("h", "hu", "hv", "z_b", "G"):
        x, y = getattr(a, f), getattr(b, f)
        assert float((x - y).abs().max()) <= 1e-12 * float(x.abs().max()), f


# the largest handler of the one-block launch and the smallest of the launches over all cells
@pytest.mark.parametrize("rows,cols", [(23, 89), (32, 64), (41, 50)])
def test_handlers_of_many_cells(rows, cols):
    """<abar_0, du_0> == <abar_N, J du_0> over 3 steps (1e-9, the bound of the other layouts) with a
    slab of rows * cols boundary cells between small handlers, one of which overwrites part of
    it."""
    from pyexner_b200.tangent import jvp_run, vjp_run
    from test_gpu_tangent import inner, tangent_state

    ny, nx = 60, 100
    arrs, params, X, Y = smooth_case(ny, nx)

    def rect(x0, x1, y0, y1):
        return [[x0 - 0.5, y0 - 0.5], [x1 + 0.5, y0 - 0.5], [x1 + 0.5, y1 + 0.5], [x0 - 0.5, y1 + 0.5]]

    spec = dict(params["boundaries"])
    spec["slab"] = dict(type="Reflective", polygon=rect(4, 3 + cols, 5, 4 + rows), values=[0.0] * 4, normal=[0.0, -1.0])
    spec["wall"] = dict(type="Transmissive", polygon=rect(6, 6, 7, 20), values=[0.0] * 4, normal=[-1.0, 0.0])
    _, cfg, mask, st = setup(arrs, dict(params, boundaries=spec), X, Y)
    assert cfg.boundaries.handlers[-2]["cells"][0].size == rows * cols
    rng = np.random.default_rng(3)
    du = tangent_state(st, rng, ("h", "hu", "hv", "z_b"))
    s, td = st.clone(), du.clone()
    jvp_run(s, td, mask, cfg, 3, "SSPRK2", 0.5)
    abar = random_adjoint(st, rng)
    rhs = inner(abar, td)
    a0 = vjp_run(st, abar.clone(), mask, cfg, 3, "SSPRK2", 0.5, checkpoint_every=2)
    assert abs(inner(a0, du, ("h", "hu", "hv", "z_b")) - rhs) <= 1e-9 * max(abs(rhs), 1e-30)

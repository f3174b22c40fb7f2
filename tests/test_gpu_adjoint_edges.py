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

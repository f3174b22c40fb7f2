"""The upper bound that lets the CFL leave faces out (re_cfl.cuh, cfl_bound), against the speeds
it bounds, pair of cells by pair of cells: called in a small kernel of their own that is compiled
like the kernels of each precision."""
import ctypes
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SOURCE = """
#include "re_cfl.cuh"
using namespace pxb;
__global__ void pairs(int m, const TYPE* x, float* bound, TYPE* fastest) {  // x: h, hu, hv, G of both cells
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    const TYPE* c = x + 8 * (size_t)k;
    const CCell<TYPE> I = make_ccell(c[0], c[1], c[2], c[3]), J = make_ccell(c[4], c[5], c[6], c[7]);
    const TYPE sx = face_speed<TYPE, false>(I, J), sy = face_speed<TYPE, true>(I, J);
    fastest[k] = nan_max(sx, sy);
    const float hi = clamp_lo((float)c[0], (float)DRY_TOL), hj = clamp_lo((float)c[4], (float)DRY_TOL);
    const float ri = f_rcp(hi), rj = f_rcp(hj);
    bound[k] = cfl_bound(fmaxf(fabsf((float)c[1]) * ri, fabsf((float)c[5]) * rj),
                         fmaxf(fabsf((float)c[2]) * ri, fabsf((float)c[6]) * rj), fmaxf(hi, hj), fminf(hi, hj),
                         fmaxf(fabsf((float)c[3]), fabsf((float)c[7])));
}
extern "C" int run_pairs(int m, const TYPE* x, float* bound, TYPE* fastest) {
    pairs<<<(m + 255) / 256, 256>>>(m, x, bound, fastest);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.parametrize("kind", ["alike", "apart", "fast", "thin", "clipped"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_bound_holds(tmp_path, dtype, kind):
    from pyexner_b200 import build

    (tmp_path / "b.cu").write_text(SOURCE.replace("TYPE", "float" if dtype == "float32" else "double"))
    so = str(tmp_path / "b.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", *(["-fmad=false"] if dtype == "float64" else []),
                    "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC, str(tmp_path / "b.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    rng = np.random.default_rng(0)
    m = 1 << 22
    # the second cell a little off the first (the bound is tight there) or anywhere
    h = 10.0 ** rng.uniform(*dict(thin=(-4.3, -2.0)).get(kind, (-2.0, 1.0)), (m, 1)) * np.ones((m, 2))
    froude = 10.0 ** rng.uniform(*dict(fast=(-0.1, 1.5), clipped=(-0.5, 0.5)).get(kind, (-3.0, -0.1)), (m, 1))
    angle = rng.uniform(0, 2 * np.pi, (m, 1)) * np.ones((m, 2))
    angle[: m // 4] = rng.choice([0.0, np.pi / 2, np.pi, 1.5 * np.pi], (m // 4, 1))  # along the axes too
    speed = froude * np.sqrt(9.81 * h[:, :1]) * np.ones((m, 2))
    G = 10.0 ** rng.uniform(*dict(clipped=(-2.0, 2.0)).get(kind, (-5.0, -1.0)), (m, 1)) * np.ones((m, 2))
    G[rng.random(m) < 0.1] = 0.0
    G[rng.random(m) < 0.1, 1] = 0.0
    if kind == "alike":
        h[:, 1] *= 1 + 1e-3 * rng.standard_normal(m)
        speed[:, 1] *= 1 + 1e-3 * rng.standard_normal(m)
    else:
        h[:, 1] *= 10.0 ** rng.uniform(-1, 1, m)
        speed[:, 1] *= rng.uniform(0, 2, m)
        angle[:, 1] = rng.uniform(0, 2 * np.pi, m)
    x = np.stack([h, h * speed * np.cos(angle), h * speed * np.sin(angle), G], axis=2).reshape(m, 8)
    xd = torch.from_numpy(np.ascontiguousarray(x.astype(dtype))).cuda()
    bound = torch.empty(m, dtype=torch.float32, device="cuda")
    fastest = torch.empty(m, dtype=xd.dtype, device="cuda")
    torch.cuda.synchronize()
    assert lib.run_pairs(m, *[ctypes.c_void_p(t.data_ptr()) for t in (xd, bound, fastest)]) == 0
    s, b = fastest.cpu().numpy().astype(np.float64), bound.cpu().numpy().astype(np.float64)
    assert np.isfinite(s).all() and np.isfinite(b).all()
    assert (s <= b).all(), float(np.max(s / b))
    if kind == "alike":  # and rules rows out: within 1 % where the cells are alike and flow along an axis
        assert np.median(b[: m // 4] / s[: m // 4]) < 1.01

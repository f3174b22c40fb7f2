"""The float64 building blocks that stand in for divisions and powers (pxb_device.cuh), called
in a small kernel of their own that is compiled like the float64 kernels."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SOURCE = """
#include "pxb_device.cuh"
__global__ void quotients(int m, const double* n, const double* d, double* q) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    const pxb::DivBy<double> by(d[k]);
    q[k] = by(n[k]);
}
__global__ void powers(int m, const double* x, double* p43, double* p32) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    p43[k] = pxb::d_pow43(x[k]);
    p32[k] = pxb::d_pow32(x[k]);
}
extern "C" int run_quotients(int m, const double* n, const double* d, double* q) {
    quotients<<<(m + 255) / 256, 256>>>(m, n, d, q);
    return (int)cudaDeviceSynchronize();
}
extern "C" int run_powers(int m, const double* x, double* p43, double* p32) {
    powers<<<(m + 255) / 256, 256>>>(m, x, p43, p32);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from pyexner_b200 import build

    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(SOURCE)
    so = str(d / "q.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    "-I", build.CSRC, str(d / "q.cu"), "-o", so], check=True)
    assert os.path.exists(so)
    return ctypes.CDLL(so)


def call(f, *arrays, outs):
    ts = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]
    rs = [torch.empty_like(ts[0]) for _ in range(outs)]
    torch.cuda.synchronize()
    assert f(len(arrays[0]), *[ctypes.c_void_p(t.data_ptr()) for t in ts + rs]) == 0
    return [r.cpu().numpy() for r in rs]


def test_quotients_are_the_division(lib):
    """The same bits for random operands of the ranges the kernels meet, for exact quotients, and
    for zeros of either sign, infinities and NaN over ordinary, zero and infinite denominators."""
    rng = np.random.default_rng(0)
    m = 1 << 22
    n = rng.standard_normal(m) * 10.0 ** rng.uniform(-30, 30, m)
    d = (1.0 + rng.random(m)) * 10.0 ** rng.uniform(-8, 8, m)
    n[: m // 8] = d[: m // 8] * rng.integers(-1000, 1000, m // 8)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, 1e-4, 3.0, -1e300])
    sn, sd = (a.ravel() for a in np.meshgrid(special, [1.0, 3.0, 1e-4, 7e5, 0.0, np.inf, np.nan]))
    n, d = np.concatenate([n, sn]), np.concatenate([d, sd])
    (q,) = call(lib.run_quotients, n, d, outs=1)
    with np.errstate(all="ignore"):
        ref = n / d
    ok = (q.view(np.int64) == ref.view(np.int64)) | (np.isnan(q) & np.isnan(ref))
    assert ok.all(), [(a, b, c, e) for a, b, c, e in zip(n[~ok], d[~ok], q[~ok], ref[~ok])][:8]


def test_subnormal_quotients_stay_within_one_step(lib):
    """Numerators so small that the remainder underflows: within one unit in the last place."""
    rng = np.random.default_rng(1)
    m = 1 << 16
    n = rng.standard_normal(m) * 10.0 ** rng.uniform(-322, -290, m)
    d = (1.0 + rng.random(m)) * 10.0 ** rng.uniform(-4, 4, m)
    (q,) = call(lib.run_quotients, n, d, outs=1)
    assert np.all(np.abs(q.view(np.int64) - (n / d).view(np.int64)) <= 1)


def test_roots_for_powers(lib):
    """Against 80-bit arithmetic: cbrt within one unit (2^-52 relative) and a product (2^-53), a
    rounded square root and a product; the second-order terms are below 1e-20."""
    rng = np.random.default_rng(2)
    x = (1.0 + rng.random(1 << 20)) * 10.0 ** rng.uniform(-8, 8, 1 << 20)
    p43, p32 = call(lib.run_powers, x, outs=2)
    xl = x.astype(np.longdouble)
    # x * cbrt(x): one Newton step on the double cube root is exact to 80 bits
    c = np.cbrt(x).astype(np.longdouble)
    c = c - (c * c * c - xl) / (3 * c * c)
    assert float(np.max(np.abs(p43 / (xl * c) - 1))) <= 1.5 * 2.0**-52 + 1e-18
    assert float(np.max(np.abs(p32 / (xl * np.sqrt(xl)) - 1))) <= 2.0**-52 + 1e-18
    z43, z32 = call(lib.run_powers, np.array([0.0, np.inf]), outs=2)
    assert z43.tolist() == [0.0, np.inf] and z32.tolist() == [0.0, np.inf]

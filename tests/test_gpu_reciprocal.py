"""The production build's reciprocal, square root and power on the GPU
(csrc/hamr_physics.cuh: rcp_nr, sqrt_nr, sqrt_nr_pos; csrc/hamr_pow.cuh), in a
small kernel compiled from the headers, against extended precision."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hamr_gamma_wind_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
KERNEL = """
#include "hamr_physics.cuh"
__global__ void k(const double *x, double *o, long n) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double rs;
    o[t] = hamr::rcp_nr(x[t]);
    o[n + t] = hamr::sqrt_nr(x[t]);
    (void)hamr::sqrt_nr_pos(x[t], rs);
    o[2 * n + t] = rs;
    o[3 * n + t] = hamr::d_pow(x[t], -13. / 9.);
}
extern "C" int run(const double *x, double *o, long n) {
    k<<<(unsigned)((n + 255) / 256), 256>>>(x, o, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("rcp")
    (d / "k.cu").write_text(KERNEL)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, str(d / "k.cu"), "-o", str(d / "k.so")], check=True)
    lib = ctypes.CDLL(str(d / "k.so"))

    def f(x):
        import torch
        xt = torch.from_numpy(np.ascontiguousarray(x, float)).cuda()
        o = torch.empty(4 * xt.numel(), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.run(ctypes.c_void_p(xt.data_ptr()), ctypes.c_void_p(o.data_ptr()), ctypes.c_long(xt.numel())) == 0
        return o.cpu().numpy().reshape(4, -1)

    return f


@pytest.mark.parametrize("span", [(-1e-6, 1e-6), (-1.0, 1.0), (-60.0, 60.0), (-300.0, 300.0)])
def test_errors_in_ulps(run, span):
    # the third-order step leaves 2^-60 (0.01 ulp) before the rounding of its
    # last sum and of the residual's product: 0.6 ulp; the root's final residual
    # less; 1/sqrt is the reciprocal of the rounded root, whose half ulp can be
    # an ulp of its reciprocal, plus half an ulp for the last sum: 1.5 ulp
    x = np.exp2(np.random.default_rng(5).uniform(*span, 400_000))
    got = run(x)
    xl = x.astype(np.longdouble)
    for q, want, bound in ((0, 1 / xl, 0.6), (1, np.sqrt(xl), 0.6), (2, 1 / np.sqrt(xl), 1.51),
                           (3, np.power(xl, np.longdouble(-13.0 / 9.0)), 0.56)):
        if q == 3 and span[1] > 60:
            continue   # beyond the normal range there: pow() itself
        ulp = np.spacing(np.abs(want.astype(float)))
        assert float(np.max(np.abs(got[q] - want) / ulp)) <= bound, q


def test_special_operands(run):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -2.0, 1e-320, 1e300, 1e-300])
    got = run(x)
    with np.errstate(all="ignore"):
        rcp, root = 1.0 / x, np.sqrt(x)
    rcp[6] = np.inf   # a subnormal operand counts as zero
    assert np.array_equal(np.isnan(got[0]), np.isnan(rcp)) and np.array_equal(got[0][:4], rcp[:4])
    assert np.isinf(got[0][6]) and np.allclose(got[0][[5, 7, 8]], rcp[[5, 7, 8]], rtol=3e-16, atol=0)
    assert np.array_equal(np.isnan(got[1]), np.isnan(root))
    ok = ~np.isnan(root)
    assert np.allclose(got[1][ok], root[ok], rtol=3e-16, atol=0)

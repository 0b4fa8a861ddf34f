"""The entropy's power function (csrc/hamr_pow.cuh) on the host, where its
fused multiply-adds round as on the GPU, against extended precision."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "hamr_gamma_wind_b200", "csrc", "hamr_pow.cuh")


@pytest.fixture(scope="module")
def pow_tab(tmp_path_factory):
    d = tmp_path_factory.mktemp("pow")
    src = d / "p.cpp"
    src.write_text(f'#include "{SRC}"\nextern "C" void f(const double *x, const double *y, double *o, long n)'
                   " { for (long k = 0; k < n; k++) o[k] = hamr::pow_tab(x[k], y[k]); }\n")
    so = d / "p.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-shared", "-fPIC", str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def f(x, y):
        x, y = np.broadcast_arrays(np.asarray(x, float), np.asarray(y, float))
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        o = np.empty_like(x)
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        lib.f(p(x), p(y), p(o), ctypes.c_long(x.size))
        return o

    return f


@pytest.mark.parametrize("gam", [13.0 / 9.0, 5.0 / 3.0, 4.0 / 3.0, 1.0 + 1e-3, 2.0])
@pytest.mark.parametrize("lo,hi", [(-1e-3, 1e-3), (-1.0, 1.0), (-70.0, 10.0), (-400.0, 400.0)])
def test_pow_error(pow_tab, gam, lo, hi):
    # half an ulp for the last sum, and before it the roundings of a term of at
    # most ln 2 / 64 = 0.011 of the result (its product and its sum with the
    # table's second word: 0.011 ulp, twice that where the result lies low in
    # its binade, the same for its argument's error), the series and the
    # logarithm below 0.01 ulp: 0.56 in all
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision on this host")
    x = np.exp2(np.random.default_rng(11).uniform(lo, hi, 200_000))
    got = pow_tab(x, -gam)
    want = np.power(x.astype(np.longdouble), np.longdouble(-gam))
    ulp = np.spacing(np.abs(want.astype(float)))
    assert float(np.max(np.abs(got - want) / ulp)) <= 0.56


def test_pow_outside_the_table(pow_tab):
    x = np.array([0.0, -0.0, -1.0, np.inf, np.nan, 5e-324, 1e-310, 1e300, 1e-300, 1.0])
    y = np.array([-1.4] * 7 + [-1.4, -1.4, -1.4])
    with np.errstate(all="ignore"):
        want = np.power(x, y)
    got = pow_tab(x, y)
    assert np.array_equal(got, want, equal_nan=True)

"""Mixed-precision steps of the face-frame solvers (HLLC, HLLD).

Their float arithmetic is ill-conditioned -- the contact speed is the
cancelling root of a quadratic -- so that a changed last bit of an edge value
or an EMF comes back as up to 1e-3 of a velocity: both answers are equally far
from FP64, but not from each other. Two things are held here:

* the arithmetic itself: one step against the values that the float kernels
  have always given (golden/mixed_face_frame.npz, recorded on a B200 from the
  production build before the PPM slopes and face values were shared; `python
  -m tests.test_gpu_mixed_face_frame OUT` records the present build's). Bound
  1e-6 of each field's norm: the FP64 parts may round differently, which on
  rare occasion turns the rounding of a value to float in one zone (measured
  up to 1e-9), while other float forms of the same formulas measured 1e-4 to
  2e-3;
* their distance from the FP64 step, over the torus body.
"""
import os
import sys

import numpy as np
import pytest

from hamr_gamma_wind_b200 import problems
from hamr_gamma_wind_b200.api import Block

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_face_frame.npz")
FIELDS = [1, 3, 5]   # u, u^2, B^1
CASES = {
    "hllc-3d": ("hllc", "ppm", (16, 12, 18)),     # metric blocks
    "hllc-3d-short": ("hllc", "ppm", (16, 12, 6)),
    "hllc-2d": ("hllc", "ppm", (40, 26, 1)),
}


def _torus(n):
    return problems.fm_torus(*n, rout=40.0, rho_atm=1e-8, u_atm=1e-10, generic=1e-3)


def _step(pb, precision, riemann, recon, steps=1):
    blk = Block(**pb.block_kwargs(), precision=precision, riemann=riemann, recon=recon)
    blk.set_geometry(pb.geo)
    blk.upload(pb.p, pb.ps)
    blk.bound()
    dt = 0.05 * min(pb.dx if pb.n3 > 1 else pb.dx[:2])
    for _ in range(steps):
        blk.step(dt)
    p, ps = blk.active(blk.download()[0]).copy(), blk.active(blk.download()[1]).copy()
    blk.close()
    return p, ps


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("rows", [False, True], ids=["faces", "rows"])
@pytest.mark.parametrize("case", list(CASES))
def test_float_face_frame_arithmetic_is_unchanged(case, rows, monkeypatch):
    if rows:
        monkeypatch.setenv("HAMR_FLUX_ROWS_MIN", "0")
    riemann, recon, n = CASES[case]
    p, _ = _step(_torus(n), "mixed", riemann, recon)
    want = np.load(GOLDEN)[case + ("-rows" if rows else "")]
    for q, k in enumerate(FIELDS):
        assert _rel(p[k], want[q]) <= 1e-6, (k, _rel(p[k], want[q]))


# four times what the step measured, over two steps (rho, u, u^1..3, B^1..3)
BODY = {
    "hllc": (1e-5, 1.3e-5, 5e-7, 3.3e-3, 4e-7, 2.5e-5, 2.5e-5, 1.2e-3),
    "hlld": (8e-5, 9e-4, 9e-5, 3.4e-2, 8e-5, 1.8e-4, 3.1e-4, 4e-3),
}


@pytest.mark.parametrize("n", [(64, 48, 32), (96, 64, 1)], ids=["3d", "2d"])
@pytest.mark.parametrize("riemann", ["hllc", "hlld"])
def test_mixed_face_frame_against_fp64(riemann, n):
    a, _ = _step(_torus(n), "mixed", riemann, "ppm", steps=2)
    b, _ = _step(_torus(n), "fp64", riemann, "ppm", steps=2)
    body = b[0] > 1e-2 * b[0].max()
    assert body.sum() > 500
    for k, bound in enumerate(BODY[riemann]):
        assert _rel(a[k][body], b[k][body]) <= bound, k


def record(path):
    """The present build's values of the first test, as the golden file holds them."""
    out = {}
    for rows in ("", "-rows"):
        if rows:
            os.environ["HAMR_FLUX_ROWS_MIN"] = "0"
        for case, (riemann, recon, n) in CASES.items():
            out[case + rows] = _step(_torus(n), "mixed", riemann, recon)[0][FIELDS]
    np.savez_compressed(path, **out)


if __name__ == "__main__":
    record(sys.argv[1])

"""A zone that is not a number: the reconstruction carries it as far as the
reference's does (the limited slope is a product with 0 or 1, which a NaN
survives), in every kernel that shares slopes and face values between zones.
One step of the strict build against the oracle: the same zones are
NaN afterwards, the others agree."""
import numpy as np
import pytest

from hamr_gamma_wind_b200 import problems
from tests._gpu import make_pair, oracle_step

pytestmark = pytest.mark.gpu

CASES = {
    "torus3d": (24, 12, 20),
    "torus2d": (33, 18, 1),
}


@pytest.mark.parametrize("rows", [False, True], ids=["faces", "rows"])
@pytest.mark.parametrize("k", [0, 2, 5])
@pytest.mark.parametrize("case", list(CASES))
def test_nan_zone_spreads_as_in_the_oracle(case, k, rows, monkeypatch):
    if rows:
        monkeypatch.setenv("HAMR_FLUX_ROWS_MIN", "0")
    pb = problems.fm_torus(*CASES[case], rout=40.0, rho_atm=1e-8, u_atm=1e-10, generic=1e-3)
    P = pb.active(pb.p)
    i, j, z = P.shape[1] // 2, P.shape[2] // 2, P.shape[3] // 2
    P[k, i, j, z] = np.nan
    blk, s = make_pair(pb)
    dt = 0.02 * min(pb.dx if pb.n3 > 1 else pb.dx[:2])
    before = np.isnan(P).any(axis=0).sum()
    blk.advance_stage(0, 0.5 * dt, dt)
    blk.advance_stage(1, dt, dt)
    oracle_step(s, dt)
    a, b = blk.active(blk.download()[0]), s.blk.active("p")
    blk.close()
    nan = np.isnan(b)
    assert nan.any(axis=0).sum() > before
    assert np.array_equal(np.isnan(a), nan)
    for q in range(9):
        ok = ~nan[q]
        assert np.abs(a[q] - b[q])[ok].max() <= 1e-13 * np.abs(b[q][ok]).max()

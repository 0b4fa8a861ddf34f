"""The merged kernels of small blocks -- both directions' fluxes with the polar
and radial rules and the centre EMFs, edge EMF with the face update, update
with the primary inversion -- against the separate kernels, bit for bit (strict
build), at sizes with remainders in every launch; and against the oracle."""
import numpy as np
import pytest

from hamr_gamma_wind_b200 import problems
from tests._gpu import field_rel_err, make_pair, oracle_step

pytestmark = pytest.mark.gpu

CASES = {
    "torus2d": lambda: problems.fm_torus(33, 17, 1, rout=40.0, rho_atm=1e-8, u_atm=1e-10),
    "torus2d-128": lambda: problems.fm_torus(128, 64, 1, rout=40.0, rho_atm=1e-8, u_atm=1e-10),
    "ot": lambda: problems.orszag_tang(31),
    "torus3d-short": lambda: problems.fm_torus(24, 13, 6, rout=40.0, rho_atm=1e-8, u_atm=1e-10),
}


def _run(pb, steps=2, **kw):
    blk, s = make_pair(pb, **kw)
    dt = 0.02 * min(pb.dx[:2] if pb.n3 == 1 else pb.dx)
    out = [blk.step(dt) for _ in range(steps)]
    return blk, s, dt, out, blk.download(), blk.download_flags()


@pytest.mark.parametrize("kw", [{}, {"recon": "mc"}, {"riemann": "hllc"}, {"inversion": "nm"}, {"floors": True}],
                         ids=["ppm", "mc", "hllc", "nm", "floors"])
@pytest.mark.parametrize("case", CASES)
def test_merged_kernels_match_separate(case, kw, monkeypatch):
    pb = CASES[case]()
    a = _run(pb, **kw)
    monkeypatch.setenv("HAMR_FLUX_ROWS_MIN", "0")   # the separate flux and EMF kernels
    monkeypatch.setenv("HAMR_CONS_INV_MAX", "0")    # the separate update and inversion
    b = _run(pb, **kw)
    assert a[3] == b[3]
    for x, y in zip(a[4] + a[5], b[4] + b[5]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("case", ["torus2d", "torus2d-128", "ot"])
def test_flat_blocks_strict(case):
    pb = CASES[case]()
    blk, s, dt, out, (p, ps), _ = _run(pb, steps=1)
    dn = oracle_step(s, dt)
    assert field_rel_err(blk, p, s, "p").max() <= 1e-14
    assert field_rel_err(blk, ps, s, "ps").max() <= 1e-14
    assert abs(out[0] - dn) <= 1e-14 * dn

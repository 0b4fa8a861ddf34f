"""The flux kernels that share slopes and face values between zones, at the
sizes where the sharing can go wrong: x3 rows that end just before, on and
after a CTA's last slot and rows shorter and longer than a CTA, and x1/x2 rows
with a remainder of one face; strict build against the oracle."""
import pytest

from hamr_gamma_wind_b200 import problems
from tests._gpu import field_rel_err, make_pair, oracle_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recon", ["ppm", "mc"])
@pytest.mark.parametrize("n3", [4, 120, 122, 124, 126, 252])
def test_x3_slots_at_cta_edges(n3, recon):
    # the bounds of the strict parity tests: PPM 1e-14 of each field's scale,
    # MC 1e-11 (more zones reach the entropy fallback, whose pow() differs in
    # the last bit)
    tol = 1e-14 if recon == "ppm" else 1e-11
    pb = problems.fm_torus(24, 10, n3, rout=40.0, rho_atm=1e-8, u_atm=1e-10)
    blk, s = make_pair(pb, recon=recon)
    dt = 0.02 * min(pb.dx)
    dn, dn_o = blk.step(dt), oracle_step(s, dt)
    p, ps = blk.download()
    assert field_rel_err(blk, p, s, "p").max() <= tol
    assert field_rel_err(blk, ps, s, "ps").max() <= tol
    assert abs(dn - dn_o) <= tol * dn_o


@pytest.mark.parametrize("recon", ["ppm", "mc"])
@pytest.mark.parametrize("n1,n2", [(24, 12), (25, 13), (35, 24)])
def test_rows_with_remainders(n1, n2, recon, monkeypatch):
    monkeypatch.setenv("HAMR_FLUX_ROWS_MIN", "0")   # rows of 12 faces also on these small blocks
    tol = 1e-14 if recon == "ppm" else 1e-11
    pb = problems.fm_torus(n1, n2, 8, rout=40.0, rho_atm=1e-8, u_atm=1e-10)
    blk, s = make_pair(pb, recon=recon)
    dt = 0.02 * min(pb.dx)
    dn, dn_o = blk.step(dt), oracle_step(s, dt)
    p, ps = blk.download()
    assert field_rel_err(blk, p, s, "p").max() <= tol
    assert field_rel_err(blk, ps, s, "ps").max() <= tol
    assert abs(dn - dn_o) <= tol * dn_o

"""Floors applied inside the bulk-copy update, after its primary inversion,
against the update followed by the separate inversion with its floors: bit for
bit (strict build), flags and failure counters included, over a row that fits
one CTA and over one cut in unequal pieces; failed zones (whose floors the
fallback pass applies) and near-vacuum zones are planted."""
import numpy as np
import pytest

from hamr_gamma_wind_b200 import problems
from hamr_gamma_wind_b200.api import Block
from tests._gpu import plant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("repair", ["none", "neighbours"])
@pytest.mark.parametrize("n3", [32, 264])
@pytest.mark.parametrize("precision,inversion", [("fp64", "2d"), ("mixed", "2d"), ("fp64", "nm")])
def test_floors_inside_update_match_separate_kernels(precision, inversion, n3, repair, monkeypatch):
    pb = problems.fm_torus(14, 9, n3, rout=40.0, rho_atm=1e-8, u_atm=1e-10)
    nfail, nthin = plant(pb)
    assert nfail > 0 and nthin > 0
    out = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("HAMR_FUSE_INV", flag)
        blk = Block(**pb.block_kwargs(), precision=precision, strict=True, inversion=inversion, floors=True,
                    repair=repair)
        blk.set_geometry(pb.geo)
        blk.upload(pb.p, pb.ps)
        blk.bound()
        dt = 0.2 * min(pb.dx)
        for _ in range(2):
            blk.advance_stage(0, 0.5 * dt, dt)
            blk.advance_stage(1, dt, dt)
        out[flag] = (*blk.download(), *blk.download_flags())
        blk.close()
    assert out["0"][3].any()
    for a, b in zip(out["1"], out["0"]):
        assert np.array_equal(a, b, equal_nan=True)

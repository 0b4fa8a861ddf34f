"""The adjoint's forward sweep, whose last segment records its steps, leaves the
objective, flags and failure counters that a sweep without records leaves:
compared with the plain forward run, bit for bit (strict build), for a last
segment that is one step, a remainder, and the whole run: on a sound torus,
whose objective is a number, and with failed zones planted so that there is
something to count (their objective may be NaN, of the same bits)."""
import numpy as np
import pytest

from hamr_gamma_wind_b200 import problems
from hamr_gamma_wind_b200.api import Adjoint, Block
from tests._gpu import plant

pytestmark = pytest.mark.gpu

STEPS = 5


def _run(call, planted):
    pb = problems.fm_torus(33, 18, 1, rout=40.0, rho_atm=1e-8, u_atm=1e-10, generic=1e-3)
    if planted:
        assert plant(pb)[0] > 0
    blk = Block(**pb.block_kwargs(), strict=True)
    blk.set_geometry(pb.geo)
    blk.upload(pb.p, pb.ps)
    blk.bound()
    adj = Adjoint(blk, pb.ng + 7)
    r = call(adj, np.full(STEPS, 0.1 * min(pb.dx[:2])))
    flags = blk.download_flags()
    adj.close()
    blk.close()
    return r, flags


@pytest.mark.parametrize("planted", [False, True], ids=["sound", "planted"])
@pytest.mark.parametrize("every", [1, 2, 3, 5, 8])
def test_recorded_sweep_leaves_the_forward_state(every, planted):
    J0, f0 = _run(lambda a, dts: a.forward(dts), planted)
    (J1, *_), f1 = _run(lambda a, dts: a.gradient(dts, every=every), planted)
    if planted:
        assert f0[1].any()
    else:
        assert np.isfinite(J0) and J0 != 0.0
    assert np.array_equal([J0], [J1], equal_nan=planted)
    for x, y in zip(f0, f1):
        assert np.array_equal(x, y)

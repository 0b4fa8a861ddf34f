"""The mixed HLL step's distance from the FP64 step over tori of several shapes
and spins, coarse ones among them, field by field. A few zones of the
atmosphere, whose energy equation is too ill-conditioned, fall to the entropy
solution in one precision and not in the other; which ones is chance, so the
worst zones of each torus are left out of its error and the events counted.

Bounds: the errors that the mixed step had before its float fluxes were
shortened, and twice its events (geometric means and sum over these tori, two
steps); measured now 0.75 to 0.86 of the errors, 18 events against 23."""
import numpy as np
import pytest

from hamr_gamma_wind_b200 import problems
from hamr_gamma_wind_b200.api import Block

pytestmark = pytest.mark.gpu

SHAPES = [(131, 77, 50), (96, 40, 26), (70, 41, 26), (64, 48, 16), (120, 64, 32), (88, 72, 40)]
# rho, u, u^1..3, B^1..3
BOUND = (6.23e-10, 4.58e-8, 7.22e-7, 1.10e-5, 5.80e-7, 5.12e-10, 8.97e-10, 2.12e-6)
EVENTS = 46   # events: zones whose internal energy is off by a tenth


def _run(pb, precision):
    blk = Block(**pb.block_kwargs(), precision=precision)
    blk.set_geometry(pb.geo)
    blk.upload(pb.p, pb.ps)
    blk.bound()
    for _ in range(2):
        blk.step(0.3 * min(pb.dx))
    p = blk.active(blk.download()[0]).reshape(9, -1)[:8].copy()
    blk.close()
    return p


def test_mixed_step_no_farther_from_fp64():
    rng = np.random.default_rng(3)
    errs, events = [], 0
    for n in SHAPES:
        pb = problems.fm_torus(*n, spin=rng.uniform(0.0, 0.98), rmax=rng.uniform(11.0, 14.0), rout=96.0, rho_atm=1e-8,
                               u_atm=1e-10, generic=1e-3, seed=int(rng.integers(1 << 20)))
        a, b = _run(pb, "mixed"), _run(pb, "fp64")
        d = np.sort(np.abs(a - b), axis=1)[:, :-max(20, a.shape[1] // 2000)]
        errs.append(np.linalg.norm(d, axis=1) / np.linalg.norm(b, axis=1))
        events += int((np.abs(a[1] - b[1]) > 0.1 * np.abs(b[1])).sum())
    gm = np.exp(np.log(np.array(errs)).mean(axis=0))
    assert (gm <= BOUND).all(), gm
    assert events <= EVENTS, events

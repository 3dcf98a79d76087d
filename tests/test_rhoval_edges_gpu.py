"""excfv_rhovalk at the edges of its tiles, against the oracle (oracle/rhoval.py).

The density kernel takes two covering points, 128 radial points and a chunk of
states per CTA, so: one harmonic (an odd number of covering points everywhere),
radial counts around 128, one state and more states than one chunk, weights
that vanish inside and at the end of the list (a vector of not-a-numbers there
must not matter), and lmaxvr above lmaxmat, where the coefficients come from the
reference layout instead of the packed one.  Each value sums the same products
as the oracle in another order: at most 2 (lmaxvr + 1)^2 of them and ngp inside
the coefficients, squared and summed, so 1e-12 of the largest entry as for the
path's other tests.
"""
import dataclasses

import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import fvref, rhoval

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmaxvr,nrmt,lradstep,nst,occupied,lmaxmat", [
    (0, 127, 1, 1, [0], 8),
    (1, 128, 1, 5, [0, 1, 3], 8),
    (2, 129, 1, 34, list(range(33)), 8),
    (4, 257, 2, 20, [0, 2, 4, 19], 8),
    (8, 131, 1, 40, list(range(0, 40, 3)), 8),
    (6, 200, 3, 12, [1, 2, 5], 3),
])
def test_density_at_the_edges(lmaxvr, nrmt, lradstep, nst, occupied, lmaxmat):
    p = syn.make_problem("diamond2", ngk=61, nstfv=nst)
    st, kp = p.static, p.kpts[0]
    rad = syn.make_radial(st, nrmt=nrmt, lmaxvr=lmaxvr)
    rng = np.random.default_rng(3)
    X = rng.standard_normal((nst, kp.nmat)) + 1j * rng.standard_normal((nst, kp.nmat))
    X = np.asfortranarray((X / np.linalg.norm(X, axis=1, keepdims=True)).T)
    wocc = np.zeros(nst)
    wocc[occupied] = rng.uniform(0.1, 2.0, len(occupied))
    zb, _, _, rf = rhoval.sht_matrices(lmaxvr) if lmaxvr else (np.full((1, 1), rhoval.lapw_math.Y00 + 0j), 0, 0,
                                                              np.full((1, 1), 1.0 / rhoval.lapw_math.Y00))
    ref = rhoval.rhovalk(st, rad, lradstep, lmaxvr, kp.ngp, fvref.match(st, kp), X, wocc, 1e-8, zb, rf)
    X[:, np.setdiff1d(np.arange(nst), occupied)] = np.nan
    with FirstVariational(0) as fv:
        fv.set_static(dataclasses.replace(st, lmaxmat=lmaxmat))
        fv.set_rho(rad, lmaxvr, lradstep, zb, rf)
        fv.rhovalk(kp, X, wocc)
        got = fv.rhomt(reset=True)
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()

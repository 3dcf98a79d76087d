"""excfv_rhovalk at the edges of its tiles, against the oracle (oracle/rhoval.py).

The density kernel takes one covering point and 128 radial points per CTA, states in
chunks of what 96 KB of shared memory hold (256 of them at lmaxvr 8 with 22 radial
functions), and atoms in groups of 64 MB of transformed states, so: one harmonic,
radial counts around 128, one state, weights that vanish inside and at the end of
the list (a vector of not-a-numbers there must not matter), lmaxvr above lmaxmat,
where the coefficients come from the reference layout instead of the packed one,
more states than one chunk, with and without spin, and more atoms than one group.
Each value sums the same products
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


def _vectors(rng, rows, cols):
    x = rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols))
    return np.asfortranarray(x / np.linalg.norm(x, axis=0))


def test_two_chunks_of_states_and_two_groups_of_atoms():
    """301 states: chunks of 256 and 45, and groups of 7 atoms and 1."""
    nst, lmaxvr = 301, 8
    p = syn.make_problem("cubic8", ngk=250, nstfv=nst, lmaxapw=8)
    st, kp = p.static, p.kpts[0]
    rad = syn.make_radial(st, nrmt=20, lmaxvr=lmaxvr)
    functions = (lmaxvr + 1) * st.apwordmax + st.nlomax
    assert 96 * 1024 // (16 * functions) < nst
    assert (64 << 20) // (16 * nst * functions * (lmaxvr + 1) ** 2) == 7 and st.natmtot == 8
    rng = np.random.default_rng(4)
    X, wocc = _vectors(rng, kp.nmat, nst), rng.uniform(0.1, 2.0, nst)
    zb, _, _, rf = rhoval.sht_matrices(lmaxvr)
    ref = rhoval.rhovalk(st, rad, 1, lmaxvr, kp.ngp, fvref.match(st, kp), X, wocc, 1e-8, zb, rf)
    with FirstVariational(0) as fv:
        fv.set_static(st)
        fv.set_rho(rad, lmaxvr, 1, zb, rf)
        fv.rhovalk(kp, X, wocc)
        got = fv.rhomt()
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()


def test_two_chunks_of_spinors():
    """Second-variational vectors of 150 states: 300 spinors in chunks of 256 and 44."""
    n, lmaxvr = 150, 8
    p = syn.make_problem("diamond2", ngk=150, nstfv=n, lmaxapw=8)
    st, kp = p.static, p.kpts[0]
    rad = syn.make_radial(st, nrmt=20, lmaxvr=lmaxvr)
    rng = np.random.default_rng(6)
    X, esv = _vectors(rng, kp.nmat, n), _vectors(rng, 2 * n, 2 * n)
    wocc = rng.uniform(0.1, 1.0, 2 * n)
    zb, _, _, rf = rhoval.sht_matrices(lmaxvr)
    rho_ref, mag_ref = rhoval.rhovalk_sv(st, rad, 1, lmaxvr, kp.ngp, fvref.match(st, kp), X, esv, wocc, 1e-8, zb, rf)
    with FirstVariational(0) as fv:
        fv.set_static(st)
        fv.set_rho(rad, lmaxvr, 1, zb, rf)
        fv.rhovalk_sv(kp, X, esv, wocc)
        rho, mag = fv.rhomt(reset=True), fv.magmt(reset=True)
    assert np.abs(rho - rho_ref).max() < 1e-12 * np.abs(rho_ref).max()
    assert np.abs(mag - mag_ref).max() < 1e-12 * np.abs(rho_ref).max()

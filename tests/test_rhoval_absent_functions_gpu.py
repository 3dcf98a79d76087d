"""The muffin-tin density where a species has fewer radial functions than the arrays.

apwfr and lofr are dimensioned for the species with the most APW orders and local
orbitals; the slots that another species does not have are never assigned, so
they may hold anything.  Two species with different apword and nlorb and an
orbital above lmaxvr, not-a-numbers in every slot that the density must not read:
the unpolarised and the spin-polarised branches against the oracle, which reads
only the functions that exist.  Bounds as in tests/test_rhoval_gpu.py.
"""
import dataclasses

import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import fvref, rhoval

pytestmark = pytest.mark.gpu


def _two_species(st):
    """Species 0: two APW orders and orbitals l = 0, 1, 3; species 1: one order, one orbital."""
    apword = np.asfortranarray(np.array([[2, 1]] * (st.lmaxapw + 1), dtype=np.int32))
    lorbl = np.asfortranarray(np.array([[0, 1], [1, 0], [3, 0]], dtype=np.int32))
    nlorb = np.array([3, 1], dtype=np.int32)
    idxlo = np.zeros((16, 3, st.natmtot), dtype=np.int32, order="F")
    i = 0
    for a in range(st.natmtot):
        for o in range(nlorb[st.idxis[a]]):
            l = int(lorbl[o, st.idxis[a]])
            for m in range(-l, l + 1):
                i += 1
                idxlo[l * (l + 1) + m, o, a] = i
    z = np.zeros
    return dataclasses.replace(
        st, apword=apword, nlomax=3, nlorb=nlorb, lorbl=lorbl, lolmax=3, idxlo=idxlo, maxnlo=11, nlotot=i,
        losize=np.array([11, 3], dtype=np.int32), loa=z((11, st.maxaa, st.natmtot), dtype=complex, order="F"),
        lolo=z((11, 11, st.natmtot), dtype=complex, order="F"), oalo=z((2, 3, st.natmtot), order="F"),
        ololo=z((3, 3, st.natmtot), order="F"), h1loa=z((2, 3, st.natmtot), order="F"),
        h1lolo=z((3, 3, st.natmtot), order="F"))


def test_absent_functions_are_not_read():
    lmaxvr, lradstep, n = 2, 2, 5
    p = syn.make_problem("cell16", ngk=65, nstfv=n, lmaxapw=4)
    st, kp = _two_species(p.static), p.kpts[0]
    rad = syn.make_radial(st, nrmt=40, lmaxvr=lmaxvr)
    rng = np.random.default_rng(5)

    def vectors(rows, cols):
        x = rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols))
        return np.asfortranarray(x / np.linalg.norm(x, axis=0))

    X, esv = vectors(kp.ngp + st.nlotot, n), vectors(2 * n, 2 * n)
    wocc, wsv = rng.uniform(0.1, 2.0, n), rng.uniform(0.1, 2.0, 2 * n)
    zb, _, _, rf = rhoval.sht_matrices(lmaxvr)
    args = (st, rad, lradstep, lmaxvr, kp.ngp, fvref.match(st, kp), X)
    ref = rhoval.rhovalk(*args, wocc, 1e-8, zb, rf)
    rho_ref, mag_ref = rhoval.rhovalk_sv(*args, esv, wsv, 1e-8, zb, rf)
    for a in range(st.natmtot):
        s = st.idxis[a]
        for l in range(st.lmaxapw + 1):
            rad.apwfr[:, :, st.apword[l, s]:, l, a] = np.nan
        rad.lofr[:, :, st.nlorb[s]:, a] = np.nan
        for o in range(st.nlorb[s]):
            if st.lorbl[o, s] > lmaxvr:
                rad.lofr[:, :, o, a] = np.nan
    assert np.isnan(rad.apwfr).any() and np.isnan(rad.lofr).any()
    with FirstVariational(0) as fv:
        fv.set_static(st)
        fv.set_rho(rad, lmaxvr, lradstep, zb, rf)
        fv.rhovalk(kp, X, wocc)
        got = fv.rhomt(reset=True)
        fv.rhovalk_sv(kp, X, esv, wsv)
        rho, mag = fv.rhomt(reset=True), fv.magmt(reset=True)
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()
    assert np.abs(rho - rho_ref).max() < 1e-12 * np.abs(rho_ref).max()
    assert np.abs(mag - mag_ref).max() < 1e-12 * np.abs(rho_ref).max()

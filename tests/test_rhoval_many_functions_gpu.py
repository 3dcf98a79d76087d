"""The muffin-tin density with very many radial functions in one launch.

700 atoms of 102 slots each, more (function, atom) pairs than a grid has rows; two
atoms of 3302 slots, more than a CTA's shared memory holds for four states.
Most slots are absent: the arrays are dimensioned by the species with the most
orbitals.  Against the oracle, bounds as in tests/test_rhoval_gpu.py.
"""
import dataclasses

import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import fvref, rhoval

pytestmark = pytest.mark.gpu


def _crowd(st, kp, copies, nlomax):
    """The cell's atoms `copies` times over, one s orbital each in arrays of nlomax slots."""
    nat = copies * st.natmtot

    def tile(x):
        return np.asfortranarray(np.tile(x, (1,) * (x.ndim - 1) + (copies,)))

    idxlo = np.zeros((1, nlomax, nat), dtype=np.int32, order="F")
    idxlo[0, 0, :] = np.arange(1, nat + 1)
    z = np.zeros
    st = dataclasses.replace(
        st, natoms=np.array([nat], dtype=np.int32), idxis=np.tile(st.idxis, copies), atposc=tile(st.atposc),
        nlomax=nlomax, nlorb=np.ones(1, dtype=np.int32), lorbl=z((nlomax, 1), dtype=np.int32, order="F"), lolmax=0,
        idxlo=idxlo, maxnlo=1, losize=np.ones(1, dtype=np.int32), nlotot=nat, aa=tile(st.aa),
        loa=z((1, st.maxaa, nat), dtype=complex, order="F"), lolo=z((1, 1, nat), dtype=complex, order="F"),
        oalo=z((st.apwordmax, nlomax, nat), order="F"), ololo=z((nlomax, nlomax, nat), order="F"),
        h1aa=tile(st.h1aa), h1loa=z((st.apwordmax, nlomax, nat), order="F"),
        h1lolo=z((nlomax, nlomax, nat), order="F"), apwfrwin=tile(st.apwfrwin))
    return st, dataclasses.replace(kp, sfacgp=tile(kp.sfacgp), nmat=kp.ngp + nat)


@pytest.mark.parametrize("copies,nlomax", [(350, 100), (1, 3300)])
def test_density(copies, nlomax):
    nst = 2 if copies > 1 else 7
    p = syn.make_problem("diamond2", ngk=61, nstfv=nst, lmaxapw=1)
    st, kp = _crowd(p.static, p.kpts[0], copies, nlomax)
    rad = syn.make_radial(st, nrmt=40, lmaxvr=0)
    rng = np.random.default_rng(copies)
    X = rng.standard_normal((kp.nmat, nst)) + 1j * rng.standard_normal((kp.nmat, nst))
    X = np.asfortranarray(X / np.linalg.norm(X, axis=0))
    wocc = rng.uniform(0.5, 2.0, nst)
    y00 = rhoval.lapw_math.Y00
    zb, rf = np.full((1, 1), y00 + 0j), np.full((1, 1), 1.0 / y00)
    ref = rhoval.rhovalk(st, rad, 1, 0, kp.ngp, fvref.match(st, kp), X, wocc, 1e-8, zb, rf)
    with FirstVariational(0) as fv:
        fv.set_static(st)
        fv.set_rho(rad, 0, 1, zb, rf)
        fv.rhovalk(kp, X, wocc)
        got = fv.rhomt()
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()

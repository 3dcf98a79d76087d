"""Matching coefficients, H and O for atoms with 5, 8 and 10 local-orbital
functions, against the oracle.

The local-orbital band takes an atom's functions eight at a time and a warp per
G+k vector, and the matching coefficients a thread per G+k vector and order: an
incomplete pass, two passes, and G+k counts that do not fill the last blocks.
Each entry is one sum of maxaa products, so 1e-13 of the largest entry as for
the path's other setups.  An orbital above lmaxapw overlaps no APW.
"""
import dataclasses

import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import fvref

pytestmark = pytest.mark.gpu


def _with_orbitals(st, ls):
    """The static with local orbitals of the given l on every atom (genidxlo's order)."""
    rng = np.random.default_rng(len(ls))
    nfun = sum(2 * l + 1 for l in ls)
    idxlo = np.zeros(((max(ls) + 1) ** 2, len(ls), st.natmtot), dtype=np.int32, order="F")
    i = 0
    for a in range(st.natmtot):
        for o, l in enumerate(ls):
            for m in range(-l, l + 1):
                i += 1
                idxlo[l * (l + 1) + m, o, a] = i
    lolo = rng.standard_normal((nfun, nfun, st.natmtot))
    ololo = rng.standard_normal((len(ls), len(ls), st.natmtot))
    return dataclasses.replace(
        st, nlomax=len(ls), nlorb=np.full(st.nspecies, len(ls), dtype=np.int32),
        lorbl=np.asfortranarray(np.tile(np.array(ls, dtype=np.int32)[:, None], (1, st.nspecies))), lolmax=max(ls),
        idxlo=idxlo, maxnlo=nfun, losize=np.full(st.nspecies, nfun, dtype=np.int32), nlotot=i,
        loa=np.asfortranarray(rng.standard_normal((nfun, st.maxaa, st.natmtot)) + 0j),
        lolo=np.asfortranarray(lolo + lolo.transpose(1, 0, 2) + 0j),
        oalo=np.asfortranarray(rng.standard_normal((st.apwordmax, len(ls), st.natmtot))),
        ololo=np.asfortranarray(ololo + ololo.transpose(1, 0, 2)),
        h1loa=np.zeros((st.apwordmax, len(ls), st.natmtot), order="F"),
        h1lolo=np.zeros((len(ls), len(ls), st.natmtot), order="F"))


@pytest.mark.parametrize("ls,ngk,shape", [((0, 0, 1), 61, "diamond2"), ((0, 0, 1, 1), 129, "cubic8"),
                                          ((1, 0, 1, 1), 100, "diamond2"), ((2, 1, 0, 1), 65, "cell16")])
def test_setup(ls, ngk, shape):
    p = syn.make_problem(shape, ngk=ngk, nstfv=4, lmaxapw=5)
    st, kp = _with_orbitals(p.static, ls), p.kpts[0]
    A = fvref.match(st, kp)
    H, O = fvref.hamiltonandoverlapsetup(st, kp, A)
    with FirstVariational(0) as fv:
        fv.set_static(st)
        got = fv.match(kp)
        assert np.abs(got - A).max() < 1e-13 * np.abs(A).max()
        h, o = fv.hamiltonandoverlapsetup(kp, got)
    up = np.triu(np.ones(H.shape, dtype=bool))
    assert np.abs(h - H)[up].max() < 1e-13 * np.abs(H).max()
    assert np.abs(o - O)[up].max() < 1e-13 * np.abs(O).max()


def test_orbital_above_lmaxapw():
    p = syn.make_problem("diamond2", ngk=61, nstfv=4, lmaxapw=2)
    st, kp = _with_orbitals(p.static, (1, 4)), p.kpts[0]
    A = fvref.match(st, kp)
    with FirstVariational(0) as fv:
        fv.set_static(st)
        h, o = fv.hamiltonandoverlapsetup(kp, fv.match(kp))
    N, nfun = kp.ngp, st.maxnlo
    for a in range(st.natmtot):
        cols = slice(N + nfun * a, N + nfun * (a + 1))
        want = np.conj(st.loa[:, :, a] @ fvref._apwi(st, A, a, N)).T
        assert np.abs(h[:N, cols] - want).max() < 1e-13 * np.abs(h).max()
        assert np.abs(o[:N, cols][:, :3]).max() > 0 and not o[:N, cols][:, 3:].any()

"""excfv_hmlint at the edges of its radial meshes and angular ranges.

The radial weights come from one tridiagonal solve and the Gaunt coefficients
from a table over |m2| = |m1 - m3|, so the smallest meshes (3 and 4 points),
meshes around a warp's 32 lanes, lmaxvr 0, and lmaxvr above lmaxmat are held to
the oracle.  A block entry sums at most (lmaxvr + 1) (nrmt + 2) products, each
rounded a few times: the bound is 4 eps times that count times the sum of the
terms' magnitudes, which the mesh's alternating spline weights keep below 30
times the largest entry.
"""
import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import mtham

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("nrmt,lmaxvr,lmaxapw,vrel", [
    (3, 2, 4, 1), (4, 4, 4, 0), (31, 0, 5, 1), (33, 3, 2, 1), (64, 6, 3, 1), (301, 8, 10, 1),
])
def test_blocks_at_the_edges(nrmt, lmaxvr, lmaxapw, vrel):
    p = syn.make_problem("diamond2", ngk=60, nstfv=6, lmaxapw=lmaxapw, valence_relativity=vrel)
    st = p.static
    st.npmatch = min(st.npmatch, nrmt)
    rad = syn.make_radial(st, nrmt=nrmt, lmaxvr=lmaxvr, sprmin=1e-2)
    aa, loa, lolo = mtham.hmlint(st, rad)
    oalo, ololo, *_ = mtham.olprad(st, rad)
    st.npmatch = max(st.apwordmax + 1, 4)
    st.sprwin = np.asfortranarray(np.linspace(1.9, 2.0, st.npmatch)[:, None] * np.ones((1, st.nspecies)))
    st.apwfrwin = np.asfortranarray(np.random.default_rng(1).uniform(
        0.5, 1.0, (st.npmatch, st.apwordmax, st.lmaxapw + 1, st.natmtot)))
    with FirstVariational(0) as fv:
        fv.set_static(st)
        first = fv.hmlint(rad)
        again = fv.hmlint(rad)     # the kept scratch holds another call's data
    tol = 4 * 2.3e-16 * (lmaxvr + 1) * (nrmt + 2) * 30
    nl = st.maxnlo
    for got in (first, again):
        for name, ref in (("aa", aa), ("loa", loa[:nl]), ("lolo", lolo[:nl, :nl]), ("oalo", oalo), ("ololo", ololo)):
            g = got[name]
            g = g[:nl] if name == "loa" else g[:nl, :nl] if name == "lolo" else g
            assert _rel(g, ref) < tol, name

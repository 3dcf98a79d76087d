"""One handle over a change of the basis (another excfv_set_static).

What a handle keeps between calls is dimensioned by the basis that it was made for.
A cell with more atoms and a larger lmaxapw, but fewer G+k vectors in arrays of the
same leading dimension, needs larger matching-coefficient arrays than the workspace
of the cell before had; single k-points and batches must get them.  The density's and
the second variation's data are refused in a basis that they do not fit, and serve on
in one that they do.  Bounds as for the path's other cells.
"""
import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from exciting_b200.lib import EXCFV_PREC_FP64, EXCFV_PREC_MIXED, ExcfvError
from oracle import fvref, rhoval

pytestmark = pytest.mark.gpu
EXCFV_ERR_STATE = -5


def _solved(shape, ngkmax, **kw):
    p = syn.make_problem(shape, nstfv=8, **kw)
    nmat = p.kpts[0].nmat
    p.kpts = [syn.make_kpoint(p.static, k.vpl, k.gkmax, ngkmax=ngkmax) for k in p.kpts]
    p.kpts[0].nmat = nmat
    refs = []
    for kp in p.kpts:
        H, O = fvref.hamiltonandoverlapsetup(p.static, kp, fvref.match(p.static, kp))
        w, _, info = fvref.solvewithlapack(H, O, p.static.nstfv, p.static.evaltol)
        assert info == 0
        refs.append((H, O, w))
    return p, refs


@pytest.mark.parametrize("prec,etol,rtol", [(EXCFV_PREC_FP64, 1e-10, 1e-13), (EXCFV_PREC_MIXED, 1e-8, 1e-7)],
                         ids=["fp64", "mixed"])
def test_workspaces_follow_the_basis(prec, etol, rtol):
    small, large = _solved("diamond2", 400, ngk=400, lmaxapw=4), _solved("cell16", 400, ngk=90, lmaxapw=8)
    n_small, n_large = small[0].nmatmax, large[0].nmatmax
    assert n_large < n_small and large[0].static.natmtot > small[0].static.natmtot
    with FirstVariational(0, precision=prec) as fv:
        fv.set_lanes(2)
        for p, refs in (small, large, small, large):
            fv.set_static(p.static)
            for kp, (H, O, w_ref) in zip(p.kpts, refs):
                w, X = fv.seceqn(kp)
                assert np.abs(w - w_ref).max() < etol
                assert fvref.residuals(H, O, w, X[:kp.nmat]).max() < rtol
            outs, info = fv.seceqn_batched(p.kpts * 3, n_small)
            assert np.all(info == 0)
            for w, _ in outs:
                assert np.abs(w - refs[0][2]).max() < etol


def test_density_and_field_data_follow_the_basis():
    lmaxvr, wocc = 2, np.array([1.0, 0.5, 0.0, 0.25, 0.75, 0.0, 0.0, 1.5])
    zb, _, _, rf = rhoval.sht_matrices(lmaxvr)

    def cell(nst):
        p = syn.make_problem("diamond2", ngk=60, nstfv=nst, lmaxapw=4)
        rad = syn.make_radial(p.static, nrmt=40, lmaxvr=lmaxvr)
        X = fvref.seceqn(p.static, p.kpts[0])[1]
        return p.static, p.kpts[0], rad, X

    with FirstVariational(0) as fv:
        for nst, fits in ((5, True), (8, False), (8, True), (4, True)):
            st, kp, rad, X = cell(nst)
            fv.set_static(st)
            if nst == 5 or (nst == 8 and fits):
                fv.set_rho(rad, lmaxvr, 1, zb, rf)
                ng, _, c = syn.make_interstitial_real(st)
                fv.set_bfield(rad, np.ones(((lmaxvr + 1) ** 2, 40, st.natmtot), order="F"), np.zeros(st.natmtot), ng,
                              np.zeros(c.shape[0]), c, 0.002)
            if fits:
                fv.rhovalk(kp, X, wocc[:nst])
                got = fv.rhomt(reset=True)
                ref = rhoval.rhovalk(st, rad, 1, lmaxvr, kp.ngp, fvref.match(st, kp), X, wocc[:nst], 1e-8, zb, rf)
                assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()
                fv.seceqnsv(kp, np.arange(nst) * 0.1, X)
                continue
            for call in (lambda: fv.rhovalk(kp, X, wocc[:nst]),
                         lambda: fv.rhovalk_sv(kp, X, np.eye(2 * nst), np.ones(2 * nst)),
                         lambda: fv.seceqnsv(kp, np.arange(nst) * 0.1, X)):
                with pytest.raises(ExcfvError) as e:
                    call()
                assert e.value.code == EXCFV_ERR_STATE

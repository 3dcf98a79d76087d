"""The dataflow panels of the tridiagonal reduction against LAPACK's ZHEGVX.

Orders where the panels' shape changes on 148 SMs, in FP64 and in complex64 storage
(odd and even leading dimensions):
  321, 352    one panel before the cluster kernel of the last columns (353: two);
  610 - 1474  block counts odd and even, a last block of one row, the workers'
              shares of tiles all in shared memory;
  1601, 1665  FP64 shares that are streamed, with a last block of one row, and
              become resident while the panels go on (complex64: from 2240);
  3201        owners with two chunks of rows, the last owner with one, and a last
              block of one row.
Two lanes of a batch have 74 SMs each, enough for the dataflow form of blocks up to
order 1024: orders 664 to 964 on two lanes at once.
Bounds as for the path's other orders.  Above 2000 the reference is a spectrum that
the matrix is built with, instead of a minute of ZHEGVX.
"""
import numpy as np
import pytest
from torch.profiler import ProfilerActivity, profile

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from exciting_b200.lib import EXCFV_PREC_FP64, EXCFV_PREC_MIXED
from oracle import fvref

pytestmark = pytest.mark.gpu


def _known_spectrum(rng, n):
    """diag(w) conjugated by six random reflectors, and w."""
    w = np.sort(rng.uniform(-1.0, 1.0, n))
    h = np.diag(rng.permutation(w)).astype(complex)
    for _ in range(6):
        v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        v /= np.linalg.norm(v)
        h -= 2.0 * np.outer(v, v.conj() @ h)
        h -= 2.0 * np.outer(h @ v, v.conj())
    return np.asfortranarray(0.5 * (h + h.conj().T)), w


@pytest.mark.parametrize("prec,n", [(EXCFV_PREC_FP64, n) for n in (321, 352, 353, 610, 641, 704, 705, 1031, 1473,
                                                                  1601, 1665, 3201)]
                         + [(EXCFV_PREC_MIXED, n) for n in (353, 827, 896, 961, 1474, 2305, 3201)])
def test_orders(prec, n):
    rng = np.random.default_rng(n)
    k = 40
    if n < 2000:
        a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        h = np.asfortranarray((a + a.conj().T) / (2 * np.sqrt(2 * n)))
        b = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        o = np.asfortranarray(np.eye(n) + 0.3 * (b @ b.conj().T) / n)
        w_ref, _, info = fvref.solvewithlapack(h.copy(), o.copy(), k, 1e-14, lwork=-1)
        assert info == 0
    else:
        h, w_ref = _known_spectrum(rng, n)
        o, w_ref = np.asfortranarray(np.eye(n, dtype=complex)), w_ref[:k]
    mixed = prec == EXCFV_PREC_MIXED
    p = syn.make_problem("diamond2", ngk=60, nstfv=6)
    with FirstVariational(0, precision=prec) as fv:
        fv.set_static(p.static)
        for _ in range(2):      # the second solve meets the first one's words
            w, x = fv.solvewithlapack(h, o, k)
            assert np.abs(w - w_ref).max() < (1e-8 if mixed else 1e-10)
            assert fvref.residuals(h, o, w, x).max() < (1e-7 if mixed else 1e-13)
            assert fvref.o_orthonormality(o, x) < (1e-9 if mixed else 1e-11)


@pytest.mark.parametrize("prec", [EXCFV_PREC_FP64, EXCFV_PREC_MIXED])
def test_two_lanes(prec):
    mixed = prec == EXCFV_PREC_MIXED
    p = syn.make_problem("cubic8", nk=4, ngk_range=(820, 900) if mixed else (600, 900), nstfv=12, lmaxapw=6)
    refs = []
    for kp in p.kpts:
        H, O = fvref.hamiltonandoverlapsetup(p.static, kp, fvref.match(p.static, kp))
        refs.append((H, O, fvref.solvewithlapack(H, O, p.static.nstfv, p.static.evaltol, lwork=-1)[0]))
    with FirstVariational(0, precision=prec) as fv:
        fv.set_static(p.static)
        fv.set_lanes(2)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            runs = [fv.seceqn_batched(p.kpts, p.nmatmax) for _ in range(3)]
    names = {e.key for e in prof.key_averages()}
    assert any("k_tridiag_flow" in n for n in names) and not any("k_tridiag_panel" in n for n in names)
    for outs, info in runs:
        assert np.all(info == 0)
        for (w, x), kp, (H, O, w_ref) in zip(outs, p.kpts, refs):
            assert np.abs(w - w_ref).max() < (1e-8 if mixed else 1e-10)
            assert fvref.residuals(H, O, w, x[:kp.nmat]).max() < (1e-7 if mixed else 1e-13)

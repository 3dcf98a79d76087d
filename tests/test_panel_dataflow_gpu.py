"""The dataflow panels of the tridiagonal reduction against LAPACK's ZHEGVX.

Orders where the panels' shape changes: one panel before the cluster kernel of
the last columns takes over, a block count that is odd or even, a last block of
one row, shares of tiles that stay in shared memory and shares that are
streamed, in FP64 and in complex64 storage (odd and even leading dimensions).
Bounds as for the path's other orders.
"""
import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from exciting_b200.lib import EXCFV_PREC_FP64, EXCFV_PREC_MIXED
from oracle import fvref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n", [(EXCFV_PREC_FP64, n) for n in (610, 641, 704, 705, 1031, 1473)]
                         + [(EXCFV_PREC_MIXED, n) for n in (827, 896, 961, 1474)])
def test_orders(prec, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    h = np.asfortranarray((a + a.conj().T) / (2 * np.sqrt(2 * n)))
    b = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    o = np.asfortranarray(np.eye(n) + 0.3 * (b @ b.conj().T) / n)
    k = 40
    w_ref, _, info = fvref.solvewithlapack(h.copy(), o.copy(), k, 1e-14, lwork=-1)
    assert info == 0
    mixed = prec == EXCFV_PREC_MIXED
    p = syn.make_problem("diamond2", ngk=60, nstfv=6)
    with FirstVariational(0, precision=prec) as fv:
        fv.set_static(p.static)
        for _ in range(2):      # the second solve meets the first one's words
            w, x = fv.solvewithlapack(h, o, k)
            assert np.abs(w - w_ref).max() < (1e-8 if mixed else 1e-10)
            assert fvref.residuals(h, o, w, x).max() < (1e-7 if mixed else 1e-13)
            assert fvref.o_orthonormality(o, x) < (1e-9 if mixed else 1e-11)

"""The eigensolve at the orders where its tiles change, against LAPACK's ZHEGVX.

The diagonal Cholesky block takes four columns per step of blocks of 64, and
products take 32 x 32 tiles with the K range in pieces where few tiles would
leave the GPU idle: orders around 4, 32, 64 and 128 and one where both tile
sizes occur, with one, few and all states wanted.  Bounds as for the path's
other orders: eigenvalues 1e-10 Ha (of matrices of norm ~1), residual 1e-13
relative, orthonormality 1e-11.

A leading minor that is not positive definite reports its order exactly as
ZPOTRF does, at every place inside a step and a block.
"""
import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import DiagonalisationFailed, FirstVariational
from oracle import fvref

pytestmark = pytest.mark.gpu


def _pair(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    h = (a + a.conj().T) / (2 * np.sqrt(2 * n))
    b = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    o = np.eye(n) + 0.3 * (b @ b.conj().T) / n
    return np.asfortranarray(h), np.asfortranarray(o)


@pytest.fixture(scope="module")
def fv():
    p = syn.make_problem("diamond2", ngk=60, nstfv=6)
    with FirstVariational(0) as f:
        f.set_static(p.static)
        yield f


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 33, 63, 64, 65, 66, 67, 127, 129, 131, 200, 333, 641])
def test_orders(fv, n):
    h, o = _pair(n, n)
    for k in sorted({1, min(n, 7), n if n <= 200 else n // 3}):
        w, x = fv.solvewithlapack(h, o, k)
        w_ref, _, info = fvref.solvewithlapack(h.copy(), o.copy(), k, 1e-14, lwork=-1)
        assert info == 0
        assert np.abs(w - w_ref).max() < 1e-10
        assert fvref.residuals(h, o, w, x).max() < 1e-13
        assert fvref.o_orthonormality(o, x) < 1e-11


@pytest.mark.parametrize("bad", [1, 2, 3, 4, 5, 31, 63, 64, 65, 66, 67, 128, 130, 131])
def test_leading_minor_not_positive_definite(fv, bad):
    n = 131
    h, o = _pair(n, 7)
    o[bad - 1, bad - 1] -= 3.0
    with pytest.raises(DiagonalisationFailed) as e:
        fv.solvewithlapack(h, o, 3)
    assert e.value.info == n + bad

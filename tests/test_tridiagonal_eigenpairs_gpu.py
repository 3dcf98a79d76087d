"""Bisection and inverse iteration on tridiagonal matrices made for their edges.

The Sturm counts run 16 leading minors at a time and fall back to pivot
quotients where the minors underflow or ||T|| is above 2^38: orders around
multiples of 16 (and of the 8 rows that inverse iteration loads at a time), zero
and tiny couplings (e^2 underflows), equal and nearly equal eigenvalues, entries
just below the limit and of 1e100, graded entries; and the numbers of states at
which the points per step change.  The matrix is passed
as H with O = 1: the reduction leaves a real tridiagonal matrix as it is.

Eigenvalues: the bisection stops at 1e-14 absolute and 2 ulp relative and the
reduction adds n roundings of ||H||, so |dw| <= 1e-14 + 8 n eps ||H||.
Residuals and orthonormality have the bounds of the path's other orders.
"""
import numpy as np
import pytest

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import fvref

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _tri(kind, n):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    d, e = rng.standard_normal(n), rng.standard_normal(max(n - 1, 0))
    if kind == "equal":
        d, e = np.full(n, 2.0), np.zeros(n - 1)
    elif kind == "split":
        e[::2] = 0.0
    elif kind == "zero diagonal":
        d, e = np.zeros(n), np.ones(n - 1)
    elif kind == "tiny couplings":
        e *= 1e-170
    elif kind == "wilkinson":
        d, e = np.abs(i - (n - 1) / 2.0), np.ones(n - 1)
    elif kind == "graded":
        d, e = 10.0 ** (-i / 4.0), 0.1 * 10.0 ** (-i[:-1] / 4.0)
    elif kind == "wide":
        d, e = d * 5e10, e * 5e10
    elif kind == "large":
        d, e = d * 1e100, e * 1e100
    return np.asfortranarray((np.diag(d) + np.diag(e, 1) + np.diag(e, -1)).astype(complex))


@pytest.fixture(scope="module")
def fv():
    p = syn.make_problem("diamond2", ngk=60, nstfv=6)
    with FirstVariational(0) as f:
        f.set_static(p.static)
        yield f


def _check(fv, h, k):
    n = h.shape[0]
    o = np.asfortranarray(np.eye(n, dtype=complex))
    w, x = fv.solvewithlapack(h, o, k)
    norm = np.abs(h).sum(axis=0).max()
    ref = np.linalg.eigvalsh(h)[:k]
    assert np.abs(w - ref).max() <= 1e-14 + 8 * n * EPS * norm
    assert (np.diff(w) >= 0).all()
    assert fvref.residuals(h, o, w, x).max() < 1e-13
    assert fvref.o_orthonormality(o, x) < 1e-11


@pytest.mark.parametrize("kind", ["random", "equal", "split", "zero diagonal", "tiny couplings", "wilkinson",
                                  "graded", "wide", "large"])
@pytest.mark.parametrize("n", [2, 9, 16, 17, 18, 33, 64, 66])
def test_edges(fv, kind, n):
    for k in sorted({1, n // 2, n}):
        _check(fv, _tri(kind, n), k)


@pytest.mark.parametrize("n,k", [(600, 100), (600, 200), (600, 400), (600, 600)])
def test_points_per_step(fv, n, k):
    _check(fv, _tri("random", n), k)

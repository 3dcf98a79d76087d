"""excfv_hmlint with local orbitals above lmaxmat, against the oracle.

The APW functions stop at lmaxmat, an atom's local orbitals may not: their Gaunt
coefficients with the APWs and with each other are wanted too.  Bound as in
tests/test_mtbuild_edges_gpu.py.
"""
import dataclasses

import numpy as np
import pytest
from test_lo_functions_gpu import _with_orbitals

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from oracle import mtham

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmaxmat,ls,lmaxvr", [(2, (0, 3, 1), 4), (1, (4, 4), 5), (0, (1, 2), 6)])
def test_blocks(lmaxmat, ls, lmaxvr):
    p = syn.make_problem("diamond2", ngk=60, nstfv=6, lmaxapw=4)
    st = dataclasses.replace(_with_orbitals(p.static, ls), lmaxmat=lmaxmat)
    nrmt = 60
    rad = syn.make_radial(st, nrmt=nrmt, lmaxvr=lmaxvr, sprmin=1e-2)
    aa, loa, lolo = mtham.hmlint(st, rad, gnt=mtham.gaunt_yry_table(max(lmaxmat, *ls), lmaxvr))
    with FirstVariational(0) as fv:
        fv.set_static(st)
        got = fv.hmlint(rad)
    tol = 4 * 2.3e-16 * (lmaxvr + 1) * (nrmt + 2) * 30
    for name, ref in (("aa", aa), ("loa", loa), ("lolo", lolo)):
        assert np.abs(got[name] - ref).max() < tol * np.abs(ref).max(), name

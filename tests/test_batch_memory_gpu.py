"""Batches when most of the device memory is taken.

A lane's workspace is sized by the caller's nmatmax.  Small orders get up to 32
lanes by default, but no more than their workspaces fit: with room for 8 lanes and
not for one per k-point the batch still runs (as it does on 8 lanes).  Where the
caller's own lane count does not fit, the call reports it and the handle goes on.
Bounds as in tests/test_batched_gpu.py.
"""
import numpy as np
import pytest
import torch

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from exciting_b200.lib import ExcfvError
from oracle import fvref

pytestmark = pytest.mark.gpu

EXCFV_ERR_ALLOC = -4
NMATMAX = 4000      # 1.2 GB for every lane
GIB = 1 << 30


@pytest.fixture(scope="module")
def small():
    p = syn.make_problem("diamond2", nk=3, ngk_range=(60, 80), nstfv=6)
    w = []
    for kp in p.kpts:
        H, O = fvref.hamiltonandoverlapsetup(p.static, kp, fvref.match(p.static, kp))
        w.append(fvref.solvewithlapack(H, O, p.static.nstfv, p.static.evaltol)[0])
    return p, w


def _fill(leave):
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info(0)[0] - leave, dtype=torch.uint8, device="cuda:0")


def test_default_lanes_fit_the_free_memory(small):
    p, w_ref = small
    with FirstVariational(0) as fv:
        fv.set_static(p.static)
        fv.seceqn(p.kpts[0])
        rest = _fill(14 * GIB)
        for _ in range(2):
            outs, info = fv.seceqn_batched(p.kpts * 10, NMATMAX)
            assert np.all(info == 0)
            assert max(np.abs(o[0] - r).max() for o, r in zip(outs, w_ref * 10)) < 1e-10
        del rest
        torch.cuda.empty_cache()
        outs, info = fv.seceqn_batched(p.kpts * 10, p.nmatmax)
        assert np.all(info == 0)
        assert max(np.abs(o[0] - r).max() for o, r in zip(outs, w_ref * 10)) < 1e-10


def test_failed_allocation_does_not_spoil_the_next_call(small):
    p, w_ref = small
    with FirstVariational(0) as fv:
        fv.set_static(p.static)
        fv.seceqn(p.kpts[0])
        fv.set_lanes(24)                    # as many as asked for, or an error
        rest = _fill(8 * GIB)
        with pytest.raises(ExcfvError) as e:
            fv.seceqn_batched(p.kpts * 8, NMATMAX)
        assert e.value.code == EXCFV_ERR_ALLOC
        assert np.abs(fv.seceqn(p.kpts[0])[0] - w_ref[0]).max() < 1e-10
        del rest
        torch.cuda.empty_cache()
        outs, info = fv.seceqn_batched(p.kpts * 8, p.nmatmax)
        assert np.all(info == 0)
        assert max(np.abs(o[0] - r).max() for o, r in zip(outs, w_ref * 8)) < 1e-10

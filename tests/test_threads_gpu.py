"""Handles of different orders driven from different host threads at the same time.

The kernels whose shared memory depends on the order (the dataflow panels, the
cluster tail, the local-orbital band, the inverse iteration) are launched by all
threads at once; a thread must not change what another thread's launch needs.
Each thread compares its results with those of the first, undisturbed solve:
sums have a fixed order, so 1e-12 (of matrices of norm ~1) is wide.
"""
import threading
import time

import numpy as np
import pytest
import torch

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational

pytestmark = pytest.mark.gpu


def _dev(a, dtype):
    return torch.from_numpy(np.asfortranarray(np.asarray(a, dtype=dtype)).ravel(order="F")).to("cuda:0")


def test_handles_of_different_orders_in_threads():
    jobs = []
    for shape, ngk in (("diamond2", 430), ("cubic8", 1300), ("diamond2", 90), ("cubic8", 700)):
        p = syn.make_problem(shape, ngk=ngk, nstfv=8, lmaxapw=6 if shape == "cubic8" else 8)
        st, kp = p.static, p.kpts[0]
        fv = FirstVariational(0)
        fv.set_static(st)
        w, _ = fv.seceqn(kp)
        t = {n: _dev(getattr(kp, n), dt) for n, dt in (("gpc", np.float64), ("tpgpc", np.float64),
                                                        ("sfacgp", np.complex128), ("igpig", np.int32),
                                                        ("vgpc", np.float64))}
        ev = torch.zeros(st.nstfv, dtype=torch.float64, device="cuda:0")
        X = torch.zeros(kp.nmat * st.nstfv, dtype=torch.complex128, device="cuda:0")
        jobs.append((fv, kp, w, t, ev, X))
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(len(jobs))

    def work(fv, kp, ref, t, ev, X):
        try:
            start.wait()
            end = time.monotonic() + 8.0
            while time.monotonic() < end and not errors:
                for _ in range(4):      # the launches of several solves ahead of the GPU
                    fv.seceqn_dev(kp.nmat, kp.ngp, kp.ngkmax, {n: x.data_ptr() for n, x in t.items()}, kp.nmat,
                                  ev.data_ptr(), X.data_ptr())
                fv.sync()
                assert np.abs(ev.cpu().numpy() - ref).max() < 1e-12
        except Exception as e:      # reported by the test below
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for fv, *_ in jobs:
        fv.close()
    assert not errors, errors

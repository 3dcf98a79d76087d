"""A captured batch never outlives what it was captured over.

Repeated device-pointer batches replay a CUDA graph whose launches carry the
addresses of the lanes' workspaces and of the status words.  Between two such
batches a host-buffer batch with larger leading dimensions makes every lane
allocate its workspace anew, and one with more k-points the status words; the
device batch must then follow the new ones.  The muffin-tin build can add the
IORA* terms of the overlap, whose launches an earlier graph does not have.  Bounds
as in tests/test_batched_gpu.py.
"""
import numpy as np
import pytest
import torch

from exciting_b200 import synthetic as syn
from exciting_b200.fv import FirstVariational
from exciting_b200.lib import EXCFV_BATCH_GROUPED, EXCFV_BATCH_LANES
from oracle import fvref

pytestmark = pytest.mark.gpu


def _dev(a, dtype):
    return torch.from_numpy(np.asfortranarray(np.asarray(a, dtype=dtype)).ravel(order="F")).to("cuda:0")


class _DeviceBatch:
    def __init__(self, fv, p):
        st = p.static
        self.fv, self.p = fv, p
        self.dk = [{n: _dev(getattr(k, n), dt) for n, dt in (
            ("gpc", np.float64), ("tpgpc", np.float64), ("sfacgp", np.complex128), ("igpig", np.int32),
            ("vgpc", np.float64))} for k in p.kpts]
        self.ev = [torch.zeros(st.nstfv, dtype=torch.float64, device="cuda:0") for _ in p.kpts]
        self.X = [torch.zeros(p.nmatmax * st.nstfv, dtype=torch.complex128, device="cuda:0") for _ in p.kpts]

    def run(self):
        p, st = self.p, self.p.static
        for e in self.ev:
            e.zero_()
        torch.cuda.synchronize()
        self.fv.seceqn_batched_dev([k.nmat for k in p.kpts], [k.ngp for k in p.kpts], p.ngkmax,
                                   *([d[n].data_ptr() for d in self.dk]
                                     for n in ("gpc", "tpgpc", "sfacgp", "igpig", "vgpc")), p.nmatmax,
                                   [e.data_ptr() for e in self.ev], [x.data_ptr() for x in self.X])
        assert np.all(self.fv.batch_info(len(p.kpts)) == 0)
        torch.cuda.synchronize()
        return [(e.cpu().numpy(), x.cpu().numpy().reshape((p.nmatmax, st.nstfv), order="F")) for e, x in
                zip(self.ev, self.X)]


def _problem(**kw):
    p = syn.make_problem("diamond2", nk=3, ngk_range=(90, 140), nstfv=8, **kw)
    refs = []
    for kp in p.kpts:
        H, O = fvref.hamiltonandoverlapsetup(p.static, kp, fvref.match(p.static, kp))
        w, _, info = fvref.solvewithlapack(H, O, p.static.nstfv, p.static.evaltol)
        assert info == 0
        refs.append((H, O, w))
    return p, refs


def _check(refs, kpts, outs):
    for (H, O, w_ref), kp, (w, X) in zip(refs, kpts, outs):
        assert np.abs(w - w_ref).max() < 1e-10
        assert fvref.residuals(H, O, w, X[:kp.nmat]).max() < 1e-13


@pytest.mark.parametrize("mode", [EXCFV_BATCH_LANES, EXCFV_BATCH_GROUPED])
def test_replay_after_the_workspaces_moved(mode):
    p, refs = _problem()
    wide = [syn.make_kpoint(p.static, k.vpl, k.gkmax, ngkmax=p.ngkmax + 50) for k in p.kpts]
    with FirstVariational(0) as fv:
        fv.set_static(p.static)
        fv.set_batch_mode(mode)
        fv.set_lanes(2)
        b = _DeviceBatch(fv, p)
        for kpts, nmatmax in ((wide, p.nmatmax + 50), (p.kpts * 2, p.nmatmax), (wide * 3, p.nmatmax + 100)):
            for _ in range(3):      # eager, captured, replayed
                _check(refs, p.kpts, b.run())
            outs, info = fv.seceqn_batched(kpts, nmatmax)
            assert np.all(info == 0)
            _check(refs * (len(kpts) // 3), p.kpts * (len(kpts) // 3), outs)
        for _ in range(3):
            _check(refs, p.kpts, b.run())


def test_replay_after_the_muffin_tin_build():
    p = syn.make_problem("diamond2", nk=3, ngk_range=(90, 140), nstfv=8, h1on=True)
    st = p.static
    st.h1aa[...], st.h1loa[...], st.h1lolo[...] = 0.0, 0.0, 0.0    # the build brings them
    rad = syn.make_radial(st, nrmt=120, lmaxvr=4)
    with FirstVariational(0) as fv:
        fv.set_static(st)
        fv.set_lanes(2)
        b = _DeviceBatch(fv, p)
        for _ in range(3):
            before = b.run()
        fv.hmlint(rad)
        refs = [fv.seceqn(kp)[0] for kp in p.kpts]
        for _ in range(3):
            after = b.run()
            for w_ref, (w, _) in zip(refs, after):
                assert np.abs(w - w_ref).max() < 1e-10
    assert max(np.abs(x[0] - y[0]).max() for x, y in zip(before, after)) > 1e-6   # the data did change

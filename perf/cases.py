"""The work that a program of this framework has it do, as cases that can be timed.

A case is one call sequence of an SCF iteration of an all-electron LAPW+lo code:

``seceqn``   one k-point from its G+k set to the lowest eigenpairs
             (``FirstVariational.seceqn`` on host buffers, as the Fortran caller
             has them, or ``seceqn_dev`` where the vectors stay on the GPU)
``kloop``    several k-points of uneven basis size in one batched call
``mtbuild``  the per-iteration operators: muffin-tin integrals and Hamiltonian
             blocks, interstitial coefficients
``secvar``   the second variation of a collinear magnet at one k-point
``density``  the muffin-tin valence density of one k-point

Eigenvectors carry an arbitrary phase, so the passes that return some fix it
(the largest component real and positive), as a program does that keeps its
vectors from one iteration to the next.

``exact`` restates each sequence in plain 64-bit NumPy and torch.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from exciting_b200 import lib as _lib
from exciting_b200 import synthetic
from exciting_b200.fv import FirstVariational

ALPHA = 1.0 / 137.03599911
Y00 = 0.5 / math.sqrt(math.pi)


def listed():
    return [
        # a primitive cell of one or two atoms at a low cutoff: the smallest k-points there are (n = 86)
        dict(name="seceqn_n86", kind="seceqn", shape="diamond2", ngk=70, nstfv=10, precision="fp64", where="host"),
        # a two-atom cell at a production cutoff (n = 316), the vectors staying on the GPU
        dict(name="seceqn_n316", kind="seceqn", shape="diamond2", ngk=300, nstfv=20, precision="fp64", where="device"),
        # an eight-atom cell at a low cutoff, an odd order (n = 715), host buffers
        dict(name="seceqn_n715", kind="seceqn", shape="cubic8", ngk=651, nstfv=60, precision="fp64", where="host"),
        # an eight-atom cell at a production cutoff (n = 1964): the configuration of the benchmark
        dict(name="seceqn_n1964", kind="seceqn", shape="cubic8", ngk=1900, nstfv=200, precision="fp64",
             where="device"),
        # the same cell in the precision form, an odd order (n = 1901) and fewer states
        dict(name="seceqn_n1901_mixed", kind="seceqn", shape="cubic8", ngk=1837, nstfv=150, precision="mixed",
             where="device"),
        # a sixteen-atom cell of two species (n = 5028): the largest single k-point
        dict(name="seceqn_n5028", kind="seceqn", shape="cell16", ngk=4900, nstfv=400, precision="fp64",
             where="device"),
        # the k-loop of a small cell: 28 k-points of n = 266..346
        dict(name="kloop_28_n300", kind="kloop", shape="diamond2", ngk_lo=250, ngk_hi=330, nk=28, nstfv=20,
             precision="fp64"),
        # the k-loop of the eight-atom cell in the precision form: 12 uneven k-points of n = 1807..2300
        dict(name="kloop_12_n2050_mixed", kind="kloop", shape="cubic8", ngk_lo=1743, ngk_hi=2236, nk=12, nstfv=200,
             precision="mixed"),
        # the operators that each iteration rebuilds from the new potential
        dict(name="mtbuild_cell8", kind="mtbuild", shape="cubic8", ngk=1900, nrmt=300, lmaxvr=8),
        # a magnetic eight-atom cell: field blocks and the two spin problems of order nstfv
        dict(name="secvar_n1964", kind="secvar", shape="cubic8", ngk=1900, nstfv=200, nrmt=250, lmaxvr=6),
        # the valence density of one k-point, about two thirds of the states occupied
        dict(name="density_n1964", kind="density", shape="cubic8", ngk=1900, nstfv=200, nocc=130, nrmt=300, lmaxvr=8,
             lradstep=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["seceqn", "seceqn", "kloop", "kloop", "mtbuild", "secvar", "density"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "seceqn":
        shape, lo, hi = rng.choice([("diamond2", 60, 340), ("cubic8", 280, 2300), ("cell16", 700, 4800)])
        ngk = _log(rng, lo, hi)
        return dict(kind=kind, shape=shape, ngk=ngk, nstfv=max(6, int(ngk * rng.uniform(0.06, 0.12))),
                    precision=precision, where="host" if ngk < 900 and rng.random() < 0.5 else "device")
    if kind == "kloop":
        shape, lo, hi, most = rng.choice([("diamond2", 60, 320, 29), ("cubic8", 300, 2000, 12)])
        ngk = _log(rng, lo, hi)
        return dict(kind=kind, shape=shape, ngk_lo=int(ngk * 0.88), ngk_hi=int(ngk * 1.1), nk=rng.randint(4, most),
                    nstfv=max(6, int(ngk * rng.uniform(0.06, 0.1))), precision=precision)
    shape, lo, hi = rng.choice([("diamond2", 80, 340), ("cubic8", 400, 1900)])
    ngk = _log(rng, lo, hi)
    lmaxvr, nrmt = rng.choice([4, 6, 8]), rng.randint(150, 400)
    if kind == "mtbuild":
        return dict(kind=kind, shape=shape, ngk=ngk, nrmt=nrmt, lmaxvr=lmaxvr)
    nstfv = max(6, int(ngk * rng.uniform(0.06, 0.11)))
    if kind == "secvar":
        return dict(kind=kind, shape=shape, ngk=ngk, nstfv=nstfv, nrmt=nrmt, lmaxvr=lmaxvr)
    return dict(kind=kind, shape=shape, ngk=ngk, nstfv=nstfv, nocc=max(2, int(nstfv * rng.uniform(0.4, 0.8))),
                nrmt=nrmt, lmaxvr=lmaxvr, lradstep=rng.choice([1, 2, 4]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _problem(case, seed):
    kw = {}
    if "ngk_lo" in case:
        kw = dict(nk=case["nk"], ngk_range=(case["ngk_lo"], case["ngk_hi"]))
    else:
        kw = dict(ngk=case["ngk"])
    if "nstfv" in case:
        kw["nstfv"] = case["nstfv"]
    # the operators' crystal is one for all seeds (its G-vector set sizes the outputs); their potential is not
    p = synthetic.make_problem(case["shape"], seed=1000 + (0 if case["kind"] == "mtbuild" else seed), **kw)
    p.nmatmax = (case["ngk_hi"] if "ngk_hi" in case else case["ngk"]) + p.static.nlotot
    return p


def _radial(case, seed, st):
    return synthetic.make_radial(st, seed=2000 + seed, nrmt=case["nrmt"], lmaxvr=case["lmaxvr"])


def _vectors(seed, rows, cols):
    """Coefficient vectors of unit length, (rows, cols) in Fortran order."""
    rng = np.random.default_rng(3000 + seed)
    x = rng.standard_normal((cols, rows)) + 1j * rng.standard_normal((cols, rows))
    return (x / np.linalg.norm(x, axis=1, keepdims=True)).T


def _pinned(a):
    """The array in page-locked memory, its values, type and Fortran order kept."""
    a = np.asarray(a)
    t = torch.empty(a.T.shape, dtype=torch.from_numpy(np.empty(0, a.dtype)).dtype,
                    pin_memory=torch.cuda.is_available())
    v = t.numpy().T
    v[...] = a
    return v


def _field(seed, st, rad):
    rng = np.random.default_rng(4000 + seed)
    lm = (rad.lmaxvr + 1) ** 2
    bxc = np.zeros((lm, rad.spr.shape[0], st.natmtot), order="F")
    for a in range(st.natmtot):
        r = rad.spr[:, int(st.idxis[a])]
        bxc[0, :, a] = (0.02 + 0.005 * rng.uniform()) * np.exp(-r) / Y00
        for q in range(1, lm):
            l = math.isqrt(q)
            bxc[q, :, a] = 0.004 * rng.standard_normal() * r ** min(l, 3) * np.exp(-r)
    return bxc, np.full(st.natmtot, 0.001)


def _spiral(n):
    """Covering points of the sphere (theta, phi)."""
    z = np.linspace(-1.0, 1.0, n)
    phi = np.zeros(n)
    for k in range(1, n - 1):
        phi[k] = phi[k - 1] + math.sqrt(8.0 * math.pi / math.sqrt(3.0) / n) / math.sqrt(1.0 - z[k] ** 2)
    return np.arccos(z), np.where(np.arange(n) == n - 1, 0.0, phi % (2.0 * math.pi))


def _real(lmax, y):
    """The real harmonics of the complex ones (points, lm)."""
    m = np.concatenate([np.arange(-l, l + 1) for l in range(lmax + 1)])
    return np.where(m == 0, y.real, math.sqrt(2.0) * np.where(m < 0, y.imag, y.real))


def _transforms(lmax):
    """Backward transform of complex harmonics and forward transform of real ones on the covering points."""
    y = _ylm(lmax, *_spiral((lmax + 1) ** 2))
    return np.asfortranarray(y), np.asfortranarray(np.linalg.inv(_real(lmax, y)))


_STREAM = []


def _stream():
    """The one stream of the program: its own work and the framework's in one order."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda()


def prepare(case, seed):
    p = _problem(case, seed)
    st = p.static
    kind = case["kind"]
    s = SimpleNamespace(case=case, p=p, st=st, kp=p.kpts[0])
    mixed = case.get("precision") == "mixed"
    s.fv = FirstVariational(0, precision=_lib.EXCFV_PREC_MIXED if mixed else _lib.EXCFV_PREC_FP64)
    if kind in ("mtbuild", "secvar", "density"):
        s.rad = _radial(case, seed, st)
    s.fv.set_static(st)
    if kind == "mtbuild":
        s.ngrid, s.veffir, s.cfunir = synthetic.make_interstitial_real(st, seed=5000 + seed)
        return s
    s.fv.reserve(p.nmatmax, p.ngkmax)
    if kind == "seceqn" and case["where"] == "host":
        s.out = (_pinned(np.zeros(st.nstfv)), _pinned(np.zeros((p.nmatmax, st.nstfv), dtype=np.complex128)))
    elif kind in ("seceqn", "kloop"):
        s.stream = _stream()
        s.fv.set_stream(s.stream.cuda_stream)
        names = ("gpc", "tpgpc", "sfacgp", "igpig", "vgpc")
        s.dev = [{n: _device(getattr(k, n)) for n in names} for k in p.kpts]
        s.eval = torch.zeros(len(p.kpts), st.nstfv, dtype=torch.float64, device="cuda")
        s.evec = torch.zeros(len(p.kpts), st.nstfv, p.nmatmax, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        cols = {n: [d[n].data_ptr() for d in s.dev] for n in names}
        if kind == "kloop":
            s.args = ([k.nmat for k in p.kpts], [k.ngp for k in p.kpts], p.ngkmax, cols["gpc"], cols["tpgpc"],
                      cols["sfacgp"], cols["igpig"], cols["vgpc"], p.nmatmax,
                      [x.data_ptr() for x in s.eval], [x.data_ptr() for x in s.evec])
        else:
            s.args = (s.kp.nmat, s.kp.ngp, p.ngkmax, {n: cols[n][0] for n in names}, p.nmatmax, s.eval.data_ptr(),
                      s.evec.data_ptr())
    elif kind == "secvar":
        s.ngrid, _, s.cfunir = synthetic.make_interstitial_real(st, seed=5000 + seed)
        s.bxc, s.bconst = _field(seed, st, s.rad)
        s.bxcir = 0.01 * np.cos(np.arange(s.cfunir.shape[0]) * 0.013)
        s.fv.set_bfield(s.rad, s.bxc, s.bconst, s.ngrid, s.bxcir, s.cfunir, 0.002)
        s.evalfv = np.sort(np.random.default_rng(6000 + seed).uniform(-0.6, 1.4, st.nstfv))
        s.evecfv = _pinned(_vectors(seed, p.nmatmax, st.nstfv))
    elif kind == "density":
        zb, rf = _transforms(case["lmaxvr"])
        s.fv.set_rho(s.rad, case["lmaxvr"], case["lradstep"], zb, rf)
        s.evecfv = _pinned(_vectors(seed, p.nmatmax, st.nstfv))
        s.wocc = np.where(np.arange(st.nstfv) < case["nocc"], 0.25, 0.0)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _fix_rows(x):
    """Each vector (last axis) with its largest component real and positive."""
    ref = x.gather(-1, x.abs().argmax(-1, keepdim=True))
    return x * (ref.conj() / ref.abs())


def _fix_columns(x):
    """The same for the columns of a NumPy array."""
    ref = x[np.abs(x).argmax(0), np.arange(x.shape[1])]
    return x * (ref.conj() / np.abs(ref))


def run(s):
    kind = s.case["kind"]
    if kind == "seceqn" and s.case["where"] == "host":
        w, x = s.fv.seceqn(s.kp, s.p.nmatmax, out=s.out)
        return w, _fix_columns(x)
    if kind in ("seceqn", "kloop"):
        with torch.cuda.stream(s.stream):
            (s.fv.seceqn_dev if kind == "seceqn" else s.fv.seceqn_batched_dev)(*s.args)
            return s.eval, _fix_rows(s.evec)
    if kind == "mtbuild":
        out = s.fv.hmlint(s.rad)
        out["veffig"] = s.fv.genveffig(s.ngrid, s.veffir, s.cfunir)
        out["meffig"] = s.fv.genmeffig(s.ngrid, s.veffir, s.cfunir)[0]
        return out
    if kind == "secvar":
        w, v = s.fv.seceqnsv(s.kp, s.evalfv, s.evecfv)
        return w, _fix_columns(v)
    s.fv.rhovalk(s.kp, s.evecfv, s.wocc)
    return s.fv.rhomt(reset=True)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

_ATOMS = {"diamond2": (2, 162), "cubic8": (8, 242), "cell16": (16, 242)}  # atoms, packed APW functions of one


def _k_work(shape, ngk, nstfv):
    na, nf = _ATOMS[shape]
    n = ngk + 8 * na
    setup = 8.0 * ngk * (ngk + 1) * na * nf + 8.0 * ngk * nf * nf * na
    eig = 32.0 / 3.0 * n ** 3 + 12.0 * n * n * nstfv
    data = 16.0 * na * nf * nf + ngk * (72.0 + 16.0 * na) + 16.0 * n * nstfv
    return data, setup + eig


def work(case):
    kind = case["kind"]
    na, nf = _ATOMS[case["shape"]]
    if kind == "seceqn":
        b, f = _k_work(case["shape"], case["ngk"], case["nstfv"])
        return {"bytes": b, "flops": f}
    if kind == "kloop":
        b, f = _k_work(case["shape"], (case["ngk_lo"] + case["ngk_hi"]) // 2, case["nstfv"])
        return {"bytes": case["nk"] * b, "flops": case["nk"] * f}
    lm = (case["lmaxvr"] + 1) ** 2
    if kind == "mtbuild":
        fn = nf // 11 * 1.0 + 4  # radial functions of an atom, about
        points = 27.0 * case["ngk"]
        return {"bytes": 8.0 * na * case["nrmt"] * (lm + 4 * fn) + 16.0 * na * (nf * nf + 8 * nf) + 64.0 * points,
                "flops": na * (2.0 * fn * fn * lm * case["nrmt"] / 2 + 4.0 * nf * nf * lm / 4)}
    n, k = case["ngk"] + 8 * na, case["nstfv"]
    if kind == "secvar":
        return {"bytes": 16.0 * (n * k + 4 * k * k + na * nf * nf) + 16.0 * case["ngk"] * na,
                "flops": na * (8.0 * case["ngk"] * nf * k + 8.0 * nf * nf * k + 8.0 * nf * k * k)
                + 8.0 * case["ngk"] ** 2 * k + 8.0 * case["ngk"] * k * k + 2 * 22.0 * k ** 3}
    nr = -(-case["nrmt"] // case["lradstep"])
    return {"bytes": 16.0 * n * k + 8.0 * na * lm * case["nrmt"],
            "flops": na * case["nocc"] * (16.0 * case["ngk"] * lm + nr * (8.0 * lm * lm + 12.0 * lm))}


def tolerance(case):
    kind = case["kind"]
    if kind in ("mtbuild", "density"):
        return {"rel": 1e-12, "max": 1e-9}
    if kind != "secvar" and case["precision"] == "mixed":
        # the vectors' first-order error of a complex64 reduction over the level spacing: 5e-7 between two runs
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-10, "max": 1e-7}  # 64-bit vectors over the level spacing: up to 5e-13 between two runs


# ---------------------------------------------------------------------------
# the same in plain 64-bit NumPy and torch
# ---------------------------------------------------------------------------

_ON = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_ON)


def _ylm(lmax, theta, phi):
    """Spherical harmonics with the Condon-Shortley phase, (points, (lmax+1)^2)."""
    c, s = np.cos(theta), np.sin(theta)
    y = np.zeros((len(theta), (lmax + 1) ** 2), dtype=np.complex128)
    pmm = np.full(len(theta), Y00)
    for m in range(lmax + 1):
        if m:
            pmm = -math.sqrt((2 * m + 1) / (2.0 * m)) * s * pmm
        below, p = np.zeros_like(pmm), pmm
        for l in range(m, lmax + 1):
            if l > m:
                a = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
                b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1))
                below, p = p, a * (c * p - b * below)
            v = p * np.exp(1j * m * phi)
            y[:, l * (l + 1) + m] = v
            y[:, l * (l + 1) - m] = (-1) ** m * v.conj()
    return y


def _bessel(lmax, x):
    """j_l(x), l = 0..lmax, by downward recurrence, (lmax+1, points)."""
    top = lmax + 40
    j = np.zeros((top + 2, len(x)))
    j[top] = 1e-200
    for l in range(top, 0, -1):
        j[l - 1] = (2 * l + 1) / x * j[l] - j[l + 1]
        j[:, np.abs(j[l - 1]) > 1e200] *= 1e-200
    j0, j1 = np.sin(x) / x, np.sin(x) / x ** 2 - np.cos(x) / x
    use0 = np.abs(j0) > np.abs(j1)
    return j[:lmax + 1] * np.where(use0, j0 / np.where(use0, j[0], 1), j1 / np.where(use0, 1, j[1]))


def _matching(st, kp):
    """Matching coefficients, (atoms, (l, m, order) packed, G+k)."""
    n, lmax, no = kp.ngp, st.lmaxapw, st.apwordmax
    y = _ylm(lmax, kp.tpgpc[0, :n], kp.tpgpc[1, :n])
    g = kp.gpc[:n]
    out = []
    for a in range(st.natmtot):
        r = float(st.rmt[st.idxis[a]])
        x = st.sprwin[:, st.idxis[a]] - r
        h = abs(x[0])
        j = _bessel(lmax + 1, g * r)
        rows = []
        for l in range(lmax + 1):
            c = np.linalg.solve(np.vander(x / h, increasing=True), st.apwfrwin[:, :, l, a])
            d = np.stack([math.factorial(q) * c[q] / h ** q for q in range(no)])
            rhs = np.stack([j[l], g * (l / (g * r) * j[l] - j[l + 1])][:no])
            sol = np.linalg.solve(d, rhs) * (4 * math.pi / math.sqrt(st.omega) * 1j ** l * kp.sfacgp[:n, a])
            for m in range(-l, l + 1):
                rows += [sol[q] * y[:, l * (l + 1) + m].conj() for q in range(no)]
        out.append(np.array(rows))
    return _t(np.array(out))


def _los(st, a):
    """(local orbital, l, m) of the atom's local-orbital functions, and the first one's row."""
    t = st.idxis[a]
    fs = [(o, int(st.lorbl[o, t]), m) for o in range(int(st.nlorb[t]))
          for m in range(-int(st.lorbl[o, t]), int(st.lorbl[o, t]) + 1)]
    o, l, m = fs[0]
    return fs, int(st.idxlo[l * (l + 1) + m, o, a]) - 1


def _matrices(st, kp):
    n, no = kp.ngp, st.apwordmax
    A = _matching(st, kp)
    H = torch.zeros(n + st.nlotot, n + st.nlotot, dtype=torch.complex128, device=_ON)
    O = torch.zeros_like(H)
    for a in range(st.natmtot):
        H[:n, :n] += A[a].mH @ (_t(st.aa[:, :, a]) @ A[a])
        O[:n, :n] += A[a].mH @ A[a]
        fs, first = _los(st, a)
        at = slice(n + first, n + first + len(fs))
        H[:n, at] = (_t(st.loa[:len(fs), :, a]) @ A[a]).mH
        H[at, at] += _t(st.lolo[:len(fs), :len(fs), a])
        for i, (o, l, m) in enumerate(fs):
            f = (l * l + l + m) * no
            O[:n, n + first + i] = (_t(st.oalo[:, o, a] + 0j) @ A[a][f:f + no]).conj()
            for i2, (o2, l2, m2) in enumerate(fs):
                if (l, m) == (l2, m2):
                    O[n + first + i, n + first + i2] += float(st.ololo[o, o2, a])
    iv = st.ivg[:, kp.igpig[:n] - 1]
    d = [_t(iv[q].astype(np.int64)) for q in range(3)]
    lo, ext = st.intgv[:, 0], st.ivgig.shape
    d = [x[:, None] - x[None, :] - int(lo[q]) for q, x in enumerate(d)]
    inside = ((d[0] >= 0) & (d[0] < ext[0]) & (d[1] >= 0) & (d[1] < ext[1]) & (d[2] >= 0) & (d[2] < ext[2]))
    flat = torch.where(inside, (d[0] * ext[1] + d[1]) * ext[2] + d[2], 0)
    ig = torch.where(inside, _t(st.ivgig.astype(np.int64)).reshape(-1)[flat], 0)
    ig = torch.where(ig <= st.ngvec, ig, 0)
    v = _t(kp.vgpc[:, :n])

    def at_g(c):
        return torch.cat([torch.zeros(1, dtype=torch.complex128, device=_ON), _t(c)])[ig]

    H[:n, :n] += at_g(st.veffig) + 0.5 * (v.T @ v) * at_g(st.meffig)
    O[:n, :n] += at_g(st.cfunig)
    return [torch.triu(M, 1) + torch.triu(M, 1).mH + torch.diag(M.diagonal().real + 0j) for M in (H, O)]


def _lowest(st, kp):
    """Eigenvalues (k) and vectors (k, n), phases fixed."""
    H, O = _matrices(st, kp)
    L = torch.linalg.cholesky(O)
    C = torch.linalg.solve_triangular(L, H, upper=False)
    C = torch.linalg.solve_triangular(L, C.mH, upper=False)
    w, z = torch.linalg.eigh(0.5 * (C + C.mH))
    x = torch.linalg.solve_triangular(L.mH, z[:, :st.nstfv], upper=True)
    return w[:st.nstfv], _fix_rows(x.T.contiguous())


def _weights(x):
    """Weights of the cubic-spline integral on the mesh x (end curvatures from the last three points)."""
    n, h = len(x), np.diff(x)
    slope = (np.eye(n)[1:] - np.eye(n)[:-1]) / h[:, None]
    M, B = np.zeros((n, n)), np.zeros((n, n))
    M[0, 0] = M[-1, -1] = 1.0
    B[0] = (slope[1] - slope[0]) / (x[2] - x[0])
    B[-1] = (slope[-1] - slope[-2]) / (x[-1] - x[-3])
    for i in range(1, n - 1):
        M[i, i - 1:i + 2] = h[i - 1] / h[i], 2 * (h[i - 1] / h[i] + 1), 1.0
        B[i] = 3 * (slope[i] - slope[i - 1]) / h[i]
    e = np.zeros(n)
    e[:-1] += h ** 3 / 12
    e[1:] += h ** 3 / 12
    w = np.zeros(n)
    w[:-1] += h / 2
    w[1:] += h / 2
    return w - np.linalg.solve(M.T, e) @ B


_GAUNT = {}


def _gaunt(lmax, lmaxvr):
    """Integrals of conj(Y_1) R_2 Y_3 over the sphere, (lm1, lm3, lm2)."""
    if (lmax, lmaxvr) not in _GAUNT:
        nt, nphi = lmax + lmaxvr // 2 + 2, 2 * lmax + lmaxvr + 3
        z, wz = np.polynomial.legendre.leggauss(nt)
        ph = 2 * math.pi * np.arange(nphi) / nphi
        th, ph = np.repeat(np.arccos(z), nphi), np.tile(ph, nt)
        wq = np.repeat(wz, nphi) * 2 * math.pi / nphi
        y, r = _ylm(lmax, th, ph), _real(lmaxvr, _ylm(lmaxvr, th, ph))
        n = y.shape[1]
        pair = (_t(y.conj() * wq[:, None])[:, :, None] * _t(y)[:, None, :]).reshape(len(wq), n * n)
        _GAUNT[lmax, lmaxvr] = (pair.T @ _t(r + 0j)).reshape(n, n, -1)
    return _GAUNT[lmax, lmaxvr]


def _blocks(st, rad, pot, kinetic):
    """aa, loa, lolo of the potential (and the kinetic energy), as the muffin-tin builder lays them out."""
    G = _gaunt(st.lmaxmat, rad.lmaxvr)
    aa = np.zeros((st.maxaa, st.maxaa, st.natmtot), dtype=np.complex128)
    loa = np.zeros((max(st.maxnlo, 1), st.maxaa, st.natmtot), dtype=np.complex128)
    lolo = np.zeros((max(st.maxnlo, 1), max(st.maxnlo, 1), st.natmtot), dtype=np.complex128)
    oalo = np.zeros((st.apwordmax, max(st.nlomax, 1), st.natmtot))
    ololo = np.zeros((max(st.nlomax, 1), max(st.nlomax, 1), st.natmtot))
    for a in range(st.natmtot):
        t = st.idxis[a]
        nr = int(rad.nrmt[t])
        x = rad.spr[:nr, t]
        w = _t(_weights(x) * x * x)
        fs = [(l, m, q) for l in range(st.lmaxmat + 1) for m in range(-l, l + 1) for q in range(st.apwordmax)]
        los, _ = _los(st, a)
        nb = (st.lmaxmat + 1) * st.apwordmax
        P = np.concatenate([rad.apwfr[:nr, 0, :, :, a].reshape(nr, -1, order="F"), rad.lofr[:nr, 0, :, a]], 1)
        D = np.concatenate([rad.apwfr[:nr, 1, :, :, a].reshape(nr, -1, order="F"), rad.lofr[:nr, 1, :, a]], 1)
        ls = np.array([b // st.apwordmax for b in range(nb)] + [int(v) for v in st.lorbl[:, t]])
        Pt, Dt = _t(P), _t(D)
        pairs = (Pt[:, :, None] * Pt[:, None, :] * w[:, None, None]).reshape(nr, -1)
        R = (pairs.T @ _t(pot[:, :nr, a].T)).reshape(P.shape[1], P.shape[1], -1)
        b = np.array([l * st.apwordmax + q for l, m, q in fs] + [nb + o for o, l, m in los])
        lm = np.array([l * l + l + m for l, m, q in fs] + [l * l + l + m for o, l, m in los])
        M = (G[lm][:, lm] * R[b][:, b]).sum(-1)
        S = (Pt * w[:, None]).T @ Pt
        if kinetic:
            av = 0.5 * ALPHA ** 2 if st.valence_relativity != 0 else 0.0
            rm = _t(1.0 / (1.0 - av * rad.veffmt[0, :nr, a] * Y00))
            K = 0.5 * ((Dt * (w * rm)[:, None]).T @ Dt) \
                + 0.5 * _t(ls * (ls + 1.0))[None, :] * ((Pt * (w * rm / _t(x * x))[:, None]).T @ Pt)
            M = M + torch.where(_t(lm)[:, None] == _t(lm)[None, :], K[b][:, b], 0.0)
        M, S = M.cpu().numpy(), S.cpu().numpy()
        nf, nl = len(fs), len(los)
        aa[:nf, :nf, a], loa[:nl, :nf, a], lolo[:nl, :nl, a] = M[:nf, :nf], M[nf:, :nf], M[nf:, nf:]
        for o in range(int(st.nlorb[t])):
            l = int(st.lorbl[o, t])
            oalo[:, o, a] = S[l * st.apwordmax:(l + 1) * st.apwordmax, nb + o]
            for o2 in range(int(st.nlorb[t])):
                if int(st.lorbl[o2, t]) == l:
                    ololo[o, o2, a] = S[nb + o, nb + o2]
    return aa, loa, lolo, oalo, ololo


def _grid_index(ngrid, iv):
    j = np.where(iv >= 0, iv, np.asarray(ngrid)[:, None] + iv).astype(np.int64)
    return j[0] + int(ngrid[0]) * (j[1] + int(ngrid[1]) * j[2])


def _at_g(st, ngrid, f):
    z = torch.fft.fftn(_t(f).reshape(tuple(int(x) for x in ngrid[::-1]))).reshape(-1) / f.shape[0]
    return z[_t(_grid_index(ngrid, st.ivg[:, :st.ngvec]))].cpu().numpy()


def _secvar(s):
    st, kp, n = s.st, s.kp, s.st.nstfv
    pot = np.array(s.bxc)
    pot[0] += s.bconst[None, :] / Y00
    aa, loa, lolo, _, _ = _blocks(st, s.rad, pot, False)
    A, E = _matching(st, kp), _t(s.evecfv)
    S = torch.zeros(n, n, dtype=torch.complex128, device=_ON)
    for a in range(st.natmtot):
        los, first = _los(st, a)
        z = A[a] @ E[:kp.ngp]
        e = E[kp.ngp + first:kp.ngp + first + len(los)]
        lz = _t(loa[:len(los), :, a])
        S += z.mH @ (_t(aa[:, :, a]) @ z + lz.T @ e) + e.mH @ (lz @ z + _t(lolo[:len(los), :len(los), a]) @ e)
    shape = tuple(int(x) for x in s.ngrid[::-1])
    at = _t(_grid_index(s.ngrid, st.ivg[:, kp.igpig[:kp.ngp] - 1]))
    g = torch.zeros(n, s.cfunir.shape[0], dtype=torch.complex128, device=_ON)
    g[:, at] = E[:kp.ngp].T
    g = torch.fft.ifftn(g.reshape(n, *shape), dim=(1, 2, 3)).reshape(n, -1) * _t((s.bxcir + 0.002) * s.cfunir)
    g = torch.fft.fftn(g.reshape(n, *shape), dim=(1, 2, 3)).reshape(n, -1)
    S += E[:kp.ngp].mH @ g[:, at].T
    w, v = np.zeros(2 * n), np.zeros((2 * n, 2 * n), dtype=np.complex128)
    for b, sign in enumerate((1.0, -1.0)):
        M = sign * S + torch.diag(_t(s.evalfv) + 0j)
        M = torch.triu(M, 1) + torch.triu(M, 1).mH + torch.diag(M.diagonal().real + 0j)
        e, z = torch.linalg.eigh(M)
        at = slice(b * n, (b + 1) * n)
        w[at], v[at, at] = e.cpu().numpy(), z.cpu().numpy()
    return w, _fix_columns(v)


def _density(s):
    st, kp, c = s.st, s.kp, s.case
    A, E = _matching(st, kp), _t(s.evecfv)[:, :c["nocc"]]
    lmax, no = c["lmaxvr"], st.apwordmax
    zb, rf = (_t(x) for x in _transforms(lmax))
    out = np.zeros(((lmax + 1) ** 2, s.rad.spr.shape[0], st.natmtot))
    ll = np.concatenate([np.full(2 * l + 1, l) for l in range(lmax + 1)])
    for a in range(st.natmtot):
        ir = np.arange(0, int(s.rad.nrmt[st.idxis[a]]), c["lradstep"])
        co = (A[a][:no * len(ll)] @ E[:kp.ngp]).reshape(len(ll), no, -1)
        u = _t(s.rad.apwfr[ir, 0, :, :, a][:, :, ll] + 0j)          # (radial, order, lm)
        los, first = _los(st, a)
        wf = torch.einsum("roq,qoj->rqj", u, co)
        for i, (o, l, m) in enumerate(los):
            if l <= lmax:
                wf[:, l * l + l + m] += _t(s.rad.lofr[ir, 0, o, a] + 0j)[:, None] * E[kp.ngp + first + i][None, :]
        f = torch.einsum("tq,rqj->rtj", zb, wf)
        f = (f.real ** 2 + f.imag ** 2) @ _t(s.wocc[:c["nocc"]])    # (radial, point)
        out[:, ir, a] = (rf @ f.T).cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    p = _problem(case, seed)
    s = SimpleNamespace(case=case, p=p, st=p.static, kp=p.kpts[0])
    if kind == "seceqn":
        w, x = _lowest(s.st, s.kp)
        return (w.cpu().numpy(), x.T.cpu().numpy()) if case["where"] == "host" else (w[None], x[None])
    if kind == "kloop":
        w = torch.zeros(len(p.kpts), s.st.nstfv, dtype=torch.float64, device=_ON)
        x = torch.zeros(len(p.kpts), s.st.nstfv, p.nmatmax, dtype=torch.complex128, device=_ON)
        for i, kp in enumerate(p.kpts):
            w[i], x[i, :, :kp.nmat] = _lowest(s.st, kp)
        return w, x
    s.rad = _radial(case, seed, s.st)
    if kind == "mtbuild":
        ngrid, v, c = synthetic.make_interstitial_real(s.st, seed=5000 + seed)
        out = dict(zip(("aa", "loa", "lolo", "oalo", "ololo"), _blocks(s.st, s.rad, s.rad.veffmt, True)))
        out["veffig"] = _at_g(s.st, ngrid, v * c)
        out["meffig"] = _at_g(s.st, ngrid, c / (1.0 - v * 0.5 * ALPHA ** 2))
        return out
    s.evecfv = _vectors(seed, p.nmatmax, s.st.nstfv)
    if kind == "secvar":
        s.ngrid, _, s.cfunir = synthetic.make_interstitial_real(s.st, seed=5000 + seed)
        s.bxc, s.bconst = _field(seed, s.st, s.rad)
        s.bxcir = 0.01 * np.cos(np.arange(s.cfunir.shape[0]) * 0.013)
        s.evalfv = np.sort(np.random.default_rng(6000 + seed).uniform(-0.6, 1.4, s.st.nstfv))
        return _secvar(s)
    s.wocc = np.where(np.arange(s.st.nstfv) < case["nocc"], 0.25, 0.0)
    return _density(s)

"""The Sturm counts of the bisection (exciting_b200/csrc/sturm.cuh), on the host.

The count at x is the number of eigenvalues of the tridiagonal matrix below x, and
rounding may move eigenvalues by a few n eps ||T||: so it lies between the exact
numbers below x - tol and x + tol.  Integer matrices at integers and halves, where
leading minors vanish exactly (also as the last but one of a run of 16, from where
the counting goes on with an infinite quotient), decoupled rows, random matrices,
and matrices above the limit of the form with minors, for orders around multiples
of 16.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "exciting_b200", "csrc")
ORDERS = [1, 2, 16, 17, 18, 19, 31, 32, 33, 34, 35, 36, 38, 39, 40, 41, 48, 49, 50, 51, 67, 120]


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("sturm") / "sturm_harness")
    subprocess.run([nvcc, "-x", "cu", "-std=c++17", "-O2", "-I", CSRC, os.path.join(HERE, "sturm_harness.cu"),
                    "-o", exe], check=True)
    return exe


def _tri(kind, n):
    rng = np.random.default_rng(n)
    d, e = np.zeros(n), np.ones(n - 1)
    if kind == "integer":
        d, e = rng.integers(-2, 3, n).astype(float), rng.integers(1, 3, n - 1).astype(float)
    elif kind == "wilkinson":
        d = np.abs(np.arange(n) - (n - 1) // 2).astype(float)
    elif kind == "decoupled":
        d, e = rng.integers(-1, 2, n).astype(float), rng.integers(0, 2, n - 1).astype(float)
    elif kind == "random":
        d, e = rng.standard_normal(n), rng.standard_normal(n - 1)
    return d, e


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 40])     # 2^40: quotients throughout
@pytest.mark.parametrize("kind", ["zero diagonal", "integer", "wilkinson", "decoupled", "random"])
def test_counts(harness, tmp_path, kind, scale):
    lines, want = [], []
    for n in ORDERS:
        d, e = _tri(kind, n)
        w = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
        norm = np.abs(d).max() + 2 * np.abs(e).max(initial=0.0)
        tol = 8 * n * np.finfo(float).eps * max(norm, 1.0)
        pivmin = np.finfo(float).tiny * max(1.0, float((scale * e).max(initial=0.0)) ** 2)
        for x in np.concatenate([np.arange(-4.0, 4.5, 0.5), w[::3], [np.sqrt(2.0), np.sqrt(3.0)]]):
            lines.append(" ".join(f"{float(v):.17g}" for v in [scale == 1.0, n, pivmin, scale * x, *(scale * d),
                                                              *(scale * e)]))
            want.append((n, x, (w < x - tol).sum(), (w < x + tol).sum()))
    inp = tmp_path / "in.txt"
    inp.write_text("\n".join(lines) + "\n")
    out = subprocess.run([harness, str(inp)], check=True, capture_output=True, text=True)
    got = [int(v) for v in out.stdout.split()]
    assert len(got) == len(want)
    wrong = [(n, x, lo, hi, g) for (n, x, lo, hi), g in zip(want, got) if not lo <= g <= hi]
    assert not wrong, wrong[:8]

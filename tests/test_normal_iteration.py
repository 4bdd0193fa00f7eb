"""The crossing normal's iteration (sym3_min_eigvec_rqi, ys_physics.cuh),
compiled for the host, against an eigenvector in extended precision.

Its result x leaves a residual r = |S x - mu x|, of which the error follows as
r / gap, the distance to the other eigenvalues. The iteration ends where the
computed residual is at most 1.8e-17 of the scale sc = sum |S_ii|, or after a
second FP64 step, which cubes an error that was below 1e-6; the computed
residual is off by up to 3 roundings of 2^-53 sc. So error times gap is at
most 3.5e-16 sc of stencils bent by up to 0.2 spacings. Rougher ones may use up
its four steps; they are accepted at a computed residual of 1e-15 sc, so 1.4e-15
sc with its roundings, else left to the Jacobi solver."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from pkg import NAME, ROOT

CSRC = os.path.join(ROOT, NAME, "csrc")

SOURCE = r"""
#include <cmath>
#include "ys_physics.cuh"
extern "C" int normals(int n, const double* S, const double* guess, double* out) {
  int done = 0;
  for (int i = 0; i < n; ++i)
    done += ys::sym3_min_eigvec_rqi(reinterpret_cast<const double(*)[3]>(S + 9 * i), guess + 3 * i, out + 3 * i);
  return done;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("normal")
    src, so = str(d / "normal.cpp"), str(d / "normal.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-w", "-fPIC", "-shared", "-ffp-contract=off",
                    "-I", CSRC, src, "-o", so, "-lm"], check=True)
    return ctypes.CDLL(so)


def _smallest(S, x):
    """The eigenvector of S's smallest eigenvalue nearest x and its gap, by
    Rayleigh-quotient iteration in extended precision (cubic: two steps from
    1e-10 are exact)."""
    S = S.astype(np.longdouble)
    x = x.astype(np.longdouble)
    for _ in range(3):
        x = x / np.sqrt((x * x).sum(1))[:, None]
        mu = np.einsum("ni,nij,nj->n", x, S, x)
        M = S - mu[:, None, None] * np.eye(3, dtype=np.longdouble)
        y = np.stack([np.cross(M[:, 1], M[:, 2]), np.cross(M[:, 2], M[:, 0]), np.cross(M[:, 0], M[:, 1])], 1)
        x = np.einsum("nij,nj->ni", y, x)
    x = x / np.sqrt((x * x).sum(1))[:, None]
    w = np.linalg.eigvalsh(S.astype(float))
    return x, w[:, 1] - w[:, 0]


def _stencils(amp, n, L=1e-3):
    rng = np.random.default_rng(1)
    p = L * np.array([[0, 0, 0], [-1, 0, 0], [1, 0, 0], [0, -1, 0], [0, 1, 0]], float)
    p = p + amp * L * rng.standard_normal((n, 5, 3))
    r = p - p.mean(1, keepdims=True)
    S = np.ascontiguousarray(np.einsum("nki,nkj->nij", r, r))
    return S, np.ascontiguousarray(np.cross(p[:, 2] - p[:, 1], p[:, 4] - p[:, 3]))


def _error(lib, S, guess):
    """error times gap over the scale of the stencils the iteration accepts,
    and how many it left to the Jacobi solver"""
    n = len(S)
    out = np.full((n, 3), np.nan)
    ptr = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    done = lib.normals(n, ptr(S), ptr(guess), ptr(out))
    ok = np.isfinite(out).all(1)
    assert ok.sum() == done
    x = out[ok].astype(np.longdouble)
    x = x / np.sqrt((x * x).sum(1))[:, None]
    v, gap = _smallest(S[ok], out[ok])
    err = np.sqrt(((x - v * (x * v).sum(1)[:, None]) ** 2).sum(1)).astype(float)
    return err * gap / np.abs(np.einsum("nii->ni", S[ok])).sum(1), n - done


@pytest.mark.parametrize("amp", [0.0, 0.02, 0.1, 0.2])
def test_residual_at_rounding(lib, amp):
    e, left = _error(lib, *_stencils(amp, 200000))
    assert left <= 100
    assert e.max() <= 3.5e-16


@pytest.mark.parametrize("amp", [0.5, 1.0])
def test_accepted_where_crumpled(lib, amp):
    e, _ = _error(lib, *_stencils(amp, 200000))
    assert e.max() <= 1.4e-15

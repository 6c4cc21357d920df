"""The fixed-point contraction of one GLL line (nekgpu_fixed.cuh) against
exact rational sums, output by output, through its test hook
nekgpu_selftest_fixed_lines.

Bound.  With U the line's largest value and d the largest entry of D, the
integers carry U in at least 2^60 units and d in at least 2^59 (the table may
give up one bit): the unit of the joined sum is at most 2^-57 U d.  Before the
last rounding an output lies within (nx + 1)/2 + sum_l |D(i,l)| / (2 d) of the
exact sum in such units (the dropped products of low limbs, D's rounding, the
join, the fields' truncation), and the last rounding adds half an ulp of the
result.

Against FP64: root mean squares over the inner and over the end outputs, no
larger than those of the FP64 multiply-add chain over the same lines.  At N=2
both round an inner output (two products by +-1/2) once; the integers' join two
bits below that adds at most 1/16 of the variance: 5 % are allowed everywhere."""
from __future__ import annotations

import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from helpers import make_ref
from nekcem_gb300 import _lib as L

LINES = 120
KINDS = ("random", "smooth", "constant", "peak", "decay", "wide")


def lines(kind, z, rng):
    n = z.size
    u = np.empty((LINES, n))
    for q in range(LINES):
        a, b = rng.standard_normal(2)
        if kind == "random":
            u[q] = rng.standard_normal(n)
        elif kind == "smooth":
            u[q] = a * np.cos(3 * rng.random() * z + 6.3 * rng.random())
        elif kind == "constant":
            u[q] = a * (1 + 1e-3 * (b * z + np.cos(3 * rng.random() * z)))
        elif kind == "peak":  # one value far above the others
            u[q] = rng.standard_normal(n) * np.where(np.arange(n) == rng.integers(n), 1.0, 1e-9)
        elif kind == "decay":
            u[q] = np.exp(-12 * (1 + 3 * rng.random()) * (z + 1)) * (1 + 0.1 * rng.standard_normal(n))
        else:  # up to 300 decades, zeros among them
            u[q] = rng.standard_normal(n) * 10.0 ** (-300 * rng.random(n)) * (rng.random(n) > 0.2)
            u[q, rng.integers(n)] = a
    return u


def matrix(N):
    ref = make_ref(N, (1, 1, 1), (0, 0, 0), (1, 1, 1), (0, 0, 0))
    n = N + 1
    D = ref.d("dxm1").copy().reshape(n, n).T  # D[i, l]
    x = ref.coords()[0][:n].copy()
    ref.close()
    return D, 2 * x - 1


def contract(D, u, split):
    n = D.shape[0]
    col = np.ascontiguousarray(D.T).reshape(-1)
    out = np.empty_like(u)
    L.check(L.load().nekgpu_selftest_fixed_lines(n, col.ctypes.data_as(L.dp), u.ctypes.data_as(L.dp),
                                                 out.ctypes.data_as(L.dp), u.shape[0], split),
            "nekgpu_selftest_fixed_lines")
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("N", [2, 3, 4, 5, 6, 7, 8])
def test_lines_against_exact_sums(N, weighted):
    D, z = matrix(N)
    n = N + 1
    if weighted:  # the reverse stage's matrix
        w = 2.0 / (N * n * np.polynomial.legendre.Legendre.basis(N)(z) ** 2)
        D = np.ascontiguousarray(D.T * w[None, :])
    F = [[Fraction(float(D[i, l])) for l in range(n)] for i in range(n)]
    d = np.abs(D).max()
    rng = np.random.default_rng(40 + N)
    for kind in KINDS:
        u = lines(kind, z, rng)
        got = contract(D, u, 0)
        np.testing.assert_array_equal(contract(D, u, 1), got)
        err = np.zeros((2, LINES, n))  # here, FP64 chain; in units of 2^-57 U d
        for q in range(LINES):
            U = Fraction(float(np.abs(u[q]).max()))
            v = [Fraction(float(x)) for x in u[q]]
            unit = U * Fraction(float(d)) / 2 ** 57
            for i in range(n):
                exact = sum(F[i][l] * v[l] for l in range(n))
                chain = 0.0
                for l in range(n):
                    chain = float(F[i][l] * v[l] + Fraction(chain))  # (rounds once)
                e = abs(Fraction(float(got[q, i])) - exact)
                bound = (n + 1) / 2 + float(np.abs(D[i]).sum()) / d / 2
                half = Fraction(float(np.spacing(abs(got[q, i])))) / 2
                assert e <= Fraction(bound) * unit + half, (kind, q, i, float(e / unit))
                err[0, q, i] = float(e / unit)
                err[1, q, i] = float(abs(Fraction(chain) - exact) / unit)
        rms = np.sqrt((err ** 2).mean(axis=1))
        for name, c in (("inner", slice(1, n - 1)), ("end", slice(0, n, n - 1))):
            here, fp64 = np.sqrt((rms[:, c] ** 2).mean(axis=1))
            assert here <= 1.05 * fp64 + 1e-6, (kind, name, here, fp64)


def test_fixed_lines_rejects_bad_arguments():
    a = np.zeros(9)
    p = a.ctypes.data_as(L.dp)
    f = L.load().nekgpu_selftest_fixed_lines
    assert f(2, p, p, p, 1, 0) == -1
    assert f(10, p, p, p, 1, 0) == -1
    assert f(3, p, p, p, 0, 0) == -1
    assert f(3, None, p, p, 1, 0) == -1
    assert f(3, p, C.cast(None, L.dp), p, 1, 0) == -1

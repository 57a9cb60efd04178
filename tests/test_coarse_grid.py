"""The coarse grids' node counts (spsim_b200/csrc/coarse_kernels.cu, restated
here): every phase a detector row can see is interpolated to 1e-8."""
import math
import os
import re

import numpy as np
import pytest


def node_count(c, t, a, fp64=False):
    cc = max(c, 1.0)
    n = 0.66 * cc + 8.9 * cc ** 0.253
    if t > 0:
        n += (3.5 + 11.5 * math.sqrt(cc / 320.0)) * t ** 1.2
    if a > 0:
        n += 6.6 * math.sqrt(a) / (1.0 + 0.5 * (cc / (8.0 * a)) ** 0.6)
    if fp64:
        n += 10.0 + cc / 100.0
    return math.ceil(n)


def interpolation(n, X):
    """Node coordinates and the barycentric interpolation matrix to X."""
    alpha = 1.0 / math.cosh(9.3 * n ** (1 / 3) / n)
    k = np.arange(n)
    xi = np.cos(np.pi * k / (n - 1))
    w = (-1.0) ** k
    w[0] *= 0.5
    w[-1] *= 0.5
    d = np.sin(math.asin(alpha) * X)[:, None] / alpha - xi[None, :]
    hit = np.abs(d) < 1e-14
    M = w / np.where(hit, 1.0, d)
    M /= M.sum(1, keepdims=True)
    rows = hit.any(1)
    M[rows] = hit[rows]
    return np.arcsin(alpha * xi) / math.asin(alpha), M


DIRS = np.array([(math.sin(p) * math.cos(q), math.sin(p) * math.sin(q), math.cos(p))
                 for p in np.linspace(0, np.pi, 7) for q in np.linspace(0, 2 * np.pi, 6, endpoint=False)])


@pytest.mark.parametrize("t", [0.05, 0.3, 0.6, 0.9, 1.2])
@pytest.mark.parametrize("c", [0.5, 3.0, 12.0, 35.0, 110.0, 260.0])
@pytest.mark.parametrize("fp64", [False, True])
def test_node_counts(c, t, fp64):
    # a row at angle atan(y) of a flat detector reaching t detector distances to
    # a side; atoms in any direction at the molecule's bound, whose phase turns
    # by c radians over half the row; with and without a falling form factor
    X = np.concatenate([np.linspace(-1, 1, 301), 1 - np.logspace(-6, -2, 30)])
    half = math.atan(t)
    R = c / half / (1.02 if t > 1 else 1.0)
    for y in (0.0, 0.5 * t, t):
        for a in (0.0, 1.0, 12.0):
            x, M = interpolation(node_count(c, t, a, fp64), X)

            def f(u):
                s = np.tan(half * u)
                rho = np.sqrt(1 + s * s + y * y)
                v = np.stack([s / rho, y / rho, 1 / rho - 1], axis=1)
                return np.exp(1j * R * (v @ DIRS.T)) * np.exp(-a * (v * v).sum(1) / t ** 2)[:, None]

            # 1e-12 beside the rounding of the phases themselves (R of them, up to 2 ulps)
            assert np.abs(M @ f(x) - f(X)).max() < (1e-12 + 4.5e-16 * R if fp64 else 1e-8), (y, a)
            # rounding errors of the nodes do not grow by more than 10 %
            assert np.sqrt((M * M).sum(1)).max() < 1.1


L = np.longdouble  # the phases' own rounding in FP64 is above 1e-15


def full_count(c, t, a, digits):
    extra = {8: 0.0, 12: 10.0 + max(c, 1.0) / 100.0, 15: 18.0 + max(c, 1.0) / 25.0}[digits]
    cc = max(c, 1.0)
    n = 0.66 * cc + 8.9 * cc ** 0.253 + (3.5 + 11.5 * math.sqrt(cc / 320.0)) * t ** 1.2 + extra
    if a > 0:
        n += 6.6 * math.sqrt(a) / (1.0 + 0.5 * (cc / (8.0 * a)) ** 0.6)
    return math.ceil(n)


@pytest.mark.parametrize("digits", [8, 12, 15])
@pytest.mark.parametrize("t", [0.02, 0.3, 0.9, 1.2])
@pytest.mark.parametrize("share", [0.0, 0.5, 0.9])
def test_node_counts_of_the_whole_range(digits, t, share):
    # every axis admitted: up to 1,024 nodes, form factors falling to e^-60, the
    # axis' middle off the beam by a share of its far end's angle
    pi = L("3.14159265358979323846264338327950288")
    X = np.concatenate([np.linspace(-1, 1, 121), 1 - np.logspace(-6, -2, 10)]).astype(L)
    dirs = DIRS[::3].astype(L)
    far = L(math.atan(t))
    mid, half = share * far, (1 - share) * far
    for c in (0.5, 2.0, 8.0, 32.0, 100.0, 320.0, 1000.0):
        for a in (0.0, 1.0, 12.0, 60.0):
            n = full_count(c, t, a, digits)
            if n > 1024:
                continue
            stretch = 9.3 * n ** (1 / 3)
            if digits == 15:
                stretch = max(stretch, 36.0)
            alpha, k = 1 / np.cosh(L(stretch / n)), np.arange(n).astype(L)
            xi = np.cos(pi * k / (n - 1))
            w = np.where(np.arange(n) & 1, L(-1), L(1))
            w[0] *= 0.5
            w[-1] *= 0.5
            d = np.sin(np.arcsin(alpha) * X)[:, None] / alpha - xi[None, :]
            hit = np.abs(d) < 1e-17
            M = w / np.where(hit, L(1), d)
            M /= M.sum(1, keepdims=True)
            M[hit.any(1)] = hit[hit.any(1)]
            R = L(c) / half / L(1.02 if t > 1 else 1.0)
            reach = np.tan(half)

            def f(u):
                s = np.tan(mid + half * u)
                rho = np.sqrt(1 + s * s)
                v = np.stack([s / rho, 0 * s, 1 / rho - 1], axis=1)
                v0 = np.array([np.sin(mid), 0, np.cos(mid) - 1])
                fall = np.exp(-L(a) * ((v - v0) ** 2).sum(1) / reach ** 2)
                return np.exp(1j * (R * (v @ dirs.T))) * fall[:, None]

            x = np.arcsin(alpha * xi) / np.arcsin(alpha)
            err = float(np.abs(M @ f(x) - f(X)).max())
            # beside eight roundings of the phases (2^-64 of R)
            assert err < 10.0 ** -digits + 8 * 2.0 ** -64 * float(R), (c, a, err)


def test_fp64_polynomials():
    # the kernels' FP64 sine, cosine and 2^x (coefficients rounded to FP64, the
    # polynomials in extended precision): to 1.7e-11 and 1e-11 for FP32 results,
    # to the rounding for FP64 ones
    header = open(os.path.join(os.path.dirname(__file__), "..", "spsim_b200", "csrc", "sincos_poly.h")).read()
    two_pi = L("6.28318530717958647692528676655900577")
    y = np.linspace(0, 0.25, 4001).astype(L)
    for name, bound in (("NODE64", 1.8e-11), ("FULL64", 2e-16)):
        for key, exact in (("S", np.sin(two_pi * y)), ("C", np.cos(two_pi * y))):
            c = re.findall(r"#define SPSIM_%s_%s\d (\S+)" % (name, key), header)
            p = np.zeros_like(y)
            for v in c[::-1]:
                p = p * y * y + L(np.float64(v))
            assert np.abs((y * p if key == "S" else p) - exact).max() < bound, (name, key)
    f = np.linspace(-0.5, 0.5, 4001).astype(L)
    for degree, bound in ((9, 1e-11), (13, 2e-16)):
        p, term = np.zeros_like(f), np.float64(1.0)
        coeffs = [term]
        for k in range(1, degree + 1):
            term = term * np.float64(0.69314718055994530942) / k
            coeffs.append(term)
        for v in coeffs[::-1]:
            p = p * f + L(v)
        assert np.abs(p / np.exp2(f) - 1).max() < bound, degree

"""The coarse grids' node counts (spsim_b200/csrc/coarse_kernels.cu, restated
here): every phase a detector row can see is interpolated to 1e-8."""
import math

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

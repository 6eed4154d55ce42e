"""The running sums of the densities take one rounding per column: their error
against extended precision stays that of a sum over the columns."""
import ctypes as C

import numpy as np
import pytest

import nuclearcgm_gb300 as ng

pytestmark = pytest.mark.gpu


def _gradient(v, ax, n, h):
    """The order-dropping first derivative along one axis in extended
    precision; v: [k][j][i][spin]."""
    v = np.moveaxis(v, ax, 0)
    g = np.zeros_like(v)
    rule = {1: [420], 2: [560, -70], 3: [630, -126, 14],
            4: [672, -168, 32, -3]}
    for i in range(n):
        if i in (0, n - 1):
            g[i] = 840 * (v[1] - v[0] if i == 0 else v[i] - v[i - 1])
            continue
        for d, c in enumerate(rule[min(i, n - 1 - i, 4)], 1):
            g[i] += c * (v[i + d] - v[i - d])
    return np.moveaxis(g / (840 * np.longdouble(h)), 0, ax)


@pytest.mark.parametrize("n,cols", [(16, 60), (17, 8)])
def test_rho_and_tau(n, cols):
    a = 0.275 * (n - 1)
    h = 2.0 * a / (n - 1)
    ax = (np.arange(n) - 0.5 * (n - 1)) * h
    z, y, x = np.meshgrid(ax, ax, ax, indexing="ij")
    rng = np.random.default_rng(n)
    X = []
    for _ in range(cols):
        o = rng.uniform(-1, 1, 3)
        g = np.exp(-((x - o[0]) ** 2 + (y - o[1]) ** 2 + (z - o[2]) ** 2) / 6)
        X.append(np.outer((g * (1 + x * rng.normal())).reshape(-1),
                          rng.normal(size=2) + 1j * rng.normal(size=2)))
    X = np.stack(X)
    ns = n ** 3
    out = [np.zeros(ns), np.zeros(ns), np.zeros(9 * ns), np.zeros(ns)]
    ctx = ng.Context(ng.Grid(n, a), cols)
    ng._check(ng.load().ncgm_densities(
        ctx.h, np.ascontiguousarray(X).ctypes.data, cols,
        *(C.c_void_p(v.ctypes.data) for v in out)))
    rho, tau = np.zeros((2, n, n, n), np.longdouble)
    for v in X.reshape(cols, n, n, n, 2):
        for part in (v.real.astype(np.longdouble),
                     v.imag.astype(np.longdouble)):
            rho += (part ** 2).sum(-1)
            for d in range(3):
                tau += (_gradient(part, d, n, h) ** 2).sum(-1)
    for got, ref in ((out[0], rho), (out[1], tau)):
        err = got - ref.reshape(-1)
        # half an ulp (2^-53 at most) of the growing sum per column, at random
        # and on average of half of the final value, and a few for a term
        assert np.sqrt((err ** 2).sum() / (ref ** 2).sum()) < (
            2.0 ** -53 * (2 + 0.5 * np.sqrt(cols / 3)))

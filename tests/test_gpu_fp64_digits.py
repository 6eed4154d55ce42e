"""The FP64 forms of ncgm_gram and ncgm_vc on the tensor cores (8 digits per
value) against extended precision: rounding-level error at the edges of the
tiles, and operands that the digit format cannot hold."""
import ctypes as C

import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi

pytestmark = pytest.mark.gpu


def _ctx(n):
    return ng.Context(ng.Grid(n, 0.5 * (n - 1) * 0.6), 4)


def _gram(ctx, A, B):
    G = np.zeros((A.shape[1], B.shape[1]), np.complex128, order="F")
    ng._check(ng.load().ncgm_gram(ctx.h, A.ctypes.data, A.shape[1],
                                  B.ctypes.data, B.shape[1], G.ctypes.data,
                                  abi.FP64))
    return G


def _vc(ctx, V, Cm):
    Y = np.zeros((V.shape[0], Cm.shape[1]), np.complex128, order="F")
    ng._check(ng.load().ncgm_vc(ctx.h, V.ctypes.data, V.shape[1],
                                Cm.ctypes.data, Cm.shape[1], Y.ctypes.data,
                                abi.FP64))
    return Y


def _block(n, p, seed):
    """Columns of very different norms, decaying away from the centre."""
    rng = np.random.default_rng(seed)
    x = np.arange(n) - 0.5 * (n - 1)
    r2 = (x[:, None, None] ** 2 + x[:, None] ** 2 + x ** 2).reshape(-1)
    env = np.repeat(np.exp(-0.15 * r2), 2)[:, None]
    A = (rng.normal(size=(2 * n ** 3, p)) +
         1j * rng.normal(size=(2 * n ** 3, p))) * env
    return np.asfortranarray(A * 10.0 ** rng.uniform(-6, 3, p))


def _pick(p):
    return sorted({0, p // 3, p // 2, p - 1})


# n = 15 is the smallest lattice of the digit form (n = 14 the plain one);
# widths around the 32- and 64-column tiles
@pytest.mark.parametrize("n,p,q", [(14, 5, 5), (15, 1, 1), (15, 32, 31),
                                   (15, 33, 64), (17, 65, 2), (16, 70, 70),
                                   (20, 130, 130)])
def test_gram(n, p, q):
    ctx = _ctx(n)
    A = _block(n, p, n + p)
    B = A if p == q else _block(n, q, n + q + 1)
    G = _gram(ctx, A, B)
    i, j = _pick(p), _pick(q)
    ref = np.array([[(A[:, a].astype(np.clongdouble).conj() *
                      B[:, b].astype(np.clongdouble)).sum() for b in j]
                    for a in i])
    scale = np.outer(np.linalg.norm(A[:, i], axis=0),
                     np.linalg.norm(B[:, j], axis=0))
    # digits beyond 2^-57 of a column's maximum, products beyond the eighth
    # level and one rounding: below 2^-51 of |a||b|
    assert (np.abs(G[np.ix_(i, j)] - ref) / scale).max() < 2.0 ** -51
    if p == q:  # a Gram of a block with itself is Hermitian to the bit
        assert np.array_equal(G, G.conj().T) or n == 14
    ctx.close()


@pytest.mark.parametrize("n,m,k", [(14, 40, 40), (15, 36, 37), (15, 100, 20),
                                   (20, 33, 32), (20, 64, 65),
                                   (17, 129, 129)])
def test_vc(n, m, k):
    ctx = _ctx(n)
    V = _block(n, m, n + m)
    rng = np.random.default_rng(m)
    s = np.abs(V).max(axis=0)
    Cm = np.asfortranarray((rng.normal(size=(m, k)) +
                            1j * rng.normal(size=(m, k))) / s[:, None])
    Y = _vc(ctx, V, Cm)
    rows = np.linspace(0, V.shape[0] - 1, 200).astype(int)
    j = _pick(k)
    ref = V[rows].astype(np.clongdouble) @ Cm[:, j].astype(np.clongdouble)
    # every row has its own scale: 2 m products, each within 2^-54 of the
    # row's largest entry times the column's
    scale = np.outer((np.abs(V[rows]) / s).max(axis=1),
                     (np.abs(Cm[:, j]) * s[:, None]).max(axis=0))
    assert (np.abs(Y[np.ix_(rows, j)] - ref) / scale).max() < (
        2 * m * 2.0 ** -54)
    ctx.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_entries(value):
    """A non-finite entry of column 3 reaches the elements that read it and
    no others."""
    n, p = 15, 40
    ctx = _ctx(n)
    A = _block(n, p, 1)
    clean = _gram(ctx, A, A), _vc(ctx, A, np.eye(p, dtype=complex, order="F"))
    A[100, 3] = value
    G, Y = _gram(ctx, A, A), _vc(ctx, A, np.eye(p, dtype=complex, order="F"))
    hit = np.zeros((p, p), bool)
    hit[3], hit[:, 3] = True, True
    assert np.array_equal(np.isfinite(G), ~hit)
    assert np.allclose(G[~hit], clean[0][~hit], rtol=1e-10, atol=0.0) or (
        np.abs(G - clean[0])[~hit].max() <= 1e-12 * np.abs(clean[0]).max())
    row = np.zeros(Y.shape, bool)
    row[100] = True  # every column of Y reads the row's entry (value * 0)
    assert np.array_equal(np.isfinite(Y), ~row)
    assert np.allclose(Y[~row], A[~row], rtol=1e-13, atol=0.0)
    ctx.close()


@pytest.mark.parametrize("scale", [1e-300, 1e280])
def test_extreme_columns(scale):
    n, p = 15, 33
    ctx = _ctx(n)
    A = _block(n, p, 2)
    A /= np.linalg.norm(A, axis=0)
    B = A.copy(order="F")
    B[:, 5] *= scale
    G, ref = _gram(ctx, A, B), _gram(ctx, A, A)
    ref[:, 5] *= scale
    assert np.abs((G - ref)[:, 5]).max() <= 1e-14 * scale
    assert np.abs(np.delete(G - ref, 5, 1)).max() <= 1e-14
    ctx.close()

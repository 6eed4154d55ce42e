"""FP64 ncgm_gram and ncgm_vc on operands where a fixed number of bits below a
column's or a row's maximum could show: nearly parallel columns, tails, nearly
triangular coefficients, columns of zeros. Against extended precision."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from test_gpu_fp64_digits import _ctx, _gram, _vc

pytestmark = pytest.mark.gpu


def _mesh(n, h):
    ax = (np.arange(n) - 0.5 * (n - 1)) * h
    z, y, x = np.meshgrid(ax, ax, ax, indexing="ij")
    return x, y, z


def _columns(n, h, w, m, seed):
    """Gaussian orbitals of width w with linear factors, unit columns."""
    x, y, z = _mesh(n, h)
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(m):
        o = rng.uniform(-2, 2, 3)
        g = np.exp(-((x - o[0]) ** 2 + (y - o[1]) ** 2 + (z - o[2]) ** 2) /
                   (2 * w * w)) * (1 + 0.3 * x + 0.2 * rng.normal() * y)
        out.append(np.outer(g.reshape(-1), rng.normal(size=2) +
                            1j * rng.normal(size=2)).reshape(-1))
    X = np.stack(out, axis=1)
    return np.asfortranarray(X / np.linalg.norm(X, axis=0))


@pytest.mark.parametrize("n,h,w", [(30, 0.55, 2.0), (24, 0.8, 2.0),
                                   (24, 0.55, 0.5)])
@pytest.mark.parametrize("eps", [1e-2, 1e-7, 1e-10])
def test_nearly_parallel_columns(n, h, w, eps):
    """Columns x and x + eps d: the products that the digits leave out have
    one sign there. The largest of them, digit 5 with itself, is below
    2^14 2^-76 of the columns' maxima per real row; roundings: one per sum of
    real products and one of their sum."""
    X, d = _columns(n, h, w, 3, 1), _columns(n, h, 1.3 * w, 3, 2)
    A = np.asfortranarray(np.concatenate([X, X + eps * d], axis=1))
    ctx = _ctx(n)
    for B in (A, A.copy(order="F")):  # digitised once, and twice
        G = _gram(ctx, A, B)
        norm, top = np.linalg.norm(A, axis=0), np.abs(A).max(axis=0)
        L = A.astype(np.clongdouble)
        for i, j in [(0, 0), (0, 3), (1, 4), (2, 5), (5, 5), (0, 1)]:
            ref = (L[:, i].conj() * L[:, j]).sum()
            left_out = 2 * A.shape[0] * 2.0 ** -62 * top[i] * top[j]
            assert abs(G[i, j] - ref) <= (2.0 ** -52 * norm[i] * norm[j] +
                                          left_out)
    ctx.close()


@pytest.mark.parametrize("n,h", [(24, 0.55), (20, 1.0)])
def test_identity_returns_the_block(n, h):
    """Y = V I: every value is held to 2^-63 of its row's largest value (both
    in units of powers of two above the columns' maxima), and rounded once."""
    x, y, z = _mesh(n, h)
    r = np.sqrt(x * x + y * y + z * z).reshape(-1)
    m = 40
    rng = np.random.default_rng(4)
    V = np.stack([np.outer(np.exp(-k * r), rng.normal(size=2) +
                           1j * rng.normal(size=2)).reshape(-1)
                  for k in np.linspace(0.4, 1.5, m)], axis=1)
    V = np.asfortranarray(V * 10.0 ** rng.uniform(-2, 2, m))
    ctx = _ctx(n)
    Y = _vc(ctx, V, np.eye(m, dtype=complex, order="F"))
    top = np.abs(V).max(axis=0)
    row = (np.abs(V) / top).max(axis=1)
    # powers of two: a factor below two for the column's and the row's scale
    bound = 2.0 ** -53 * np.abs(V) + 4 * 2.0 ** -63 * np.outer(row, top)
    assert (np.abs(Y.real - V.real) <= bound).all()
    assert (np.abs(Y.imag - V.imag) <= bound).all()
    ctx.close()


def test_nearly_triangular_coefficients():
    """V R^-1 of the orthonormalisation: one product dominates each sum, and
    the result is rounded to within its own rounding."""
    n, m = 24, 60
    V = _columns(n, 0.55, 2.0, m, 5)
    Cm = np.triu(np.eye(m) + 0.01 * np.random.default_rng(6).normal(
        size=(m, m))) + 0j
    Y = _vc(_ctx(n), V, np.asfortranarray(Cm))
    rows = np.linspace(0, V.shape[0] - 1, 1500).astype(int)
    ref = V[rows].astype(np.clongdouble) @ Cm.astype(np.clongdouble)
    err = np.abs(Y[rows] - ref)
    assert np.sqrt((err ** 2).sum() / (np.abs(ref) ** 2).sum()) < 2.0 ** -53


def test_column_of_zeros():
    """Coefficients of a column of zeros do not set the scale of the others."""
    n, m = 20, 40
    V = _columns(n, 0.6, 1.5, m, 7)
    V[:, 3] = 0.0
    V[:, 5].real = 0.0
    rng = np.random.default_rng(8)
    Cm = np.asfortranarray(rng.normal(size=(m, m)) +
                           1j * rng.normal(size=(m, m)))
    clean = _vc(_ctx(n), V, Cm)
    Cm[3] *= 1e30
    Y = _vc(_ctx(n), V, Cm)
    assert np.abs(Y - clean).max() <= 2.0 ** -52 * np.abs(clean).max()

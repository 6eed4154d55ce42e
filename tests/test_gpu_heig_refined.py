"""The FP64 projected eigensolver between its size limits (48 <= m <= 80): the
double-float stage, its FP64 refinement and the cluster rotations, against
numpy, on spectra that reach each of them, and the inputs it hands back to the
Jacobi method."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi

pytestmark = pytest.mark.gpu


def _unitary(m, rng):
    return np.linalg.qr(rng.normal(size=(m, m)) +
                        1j * rng.normal(size=(m, m)))[0]


def _matrix(kind, m, rng):
    Q = _unitary(m, rng)
    if kind == "generic":
        w = rng.normal(size=m)
    elif kind == "kramers":  # exact pairs up to the rounding of the product
        w = np.repeat(np.sort(rng.normal(size=(m + 1) // 2)), 2)[:m]
    elif kind == "occupations":  # two clusters with gaps down to 1e-14
        w = np.where(np.arange(m) < m // 2, 10.0 ** -rng.uniform(3, 14, m),
                     1 - 10.0 ** -rng.uniform(3, 14, m))
    elif kind == "close":  # gaps on both sides of the cluster rule
        w = np.cumsum(10.0 ** rng.uniform(-9, 0, m))
    elif kind == "graded":
        w = 10.0 ** rng.uniform(-12, 3, m) * rng.choice([-1, 1], m)
    elif kind == "unit":
        w = np.full(m, -3.5)
    elif kind == "large":
        w = rng.normal(size=m) * 2.0 ** 700
    else:
        w = rng.normal(size=m) * 2.0 ** -700
    A = (Q * w) @ Q.conj().T
    A = 0.5 * (A + A.conj().T)
    return np.asfortranarray(A)


def _heig(A):
    m = A.shape[0]
    ctx = ng.Context(ng.Grid(8, 3.0), 2)
    w = np.zeros(m)
    V = np.zeros((m, m), np.complex128, order="F")
    rc = ng.load().ncgm_heig(ctx.h, A.ctypes.data, m, w.ctypes.data,
                             V.ctypes.data, abi.FP64)
    ctx.close()
    return rc, w, V


@pytest.mark.parametrize("kind", ["generic", "kramers", "occupations", "close",
                                  "graded", "unit", "large", "small"])
@pytest.mark.parametrize("m", [48, 63, 80])
def test_refined_eigensolver(m, kind):
    """Each entry of X^H X and X^H A X is a sum of at most 2 m products and
    carries their roundings, 2 m eps in all; the same bound holds numpy's."""
    A = _matrix(kind, m, np.random.default_rng(m))
    rc, w, V = _heig(A)
    assert rc == 0
    ref = np.linalg.eigvalsh(A)
    scale = np.abs(ref).max()
    tol = 2 * m * 2.3e-16
    assert (np.diff(w) >= 0).all()
    assert np.abs(w - ref).max() / scale <= tol
    assert np.abs(V.conj().T @ V - np.eye(m)).max() <= tol
    assert np.abs((A / scale) @ V - V * (w / scale)).max() <= tol


def test_handed_back():
    """A zero matrix and a diagonal one keep their results; one with a NaN
    still reports that it did not converge."""
    m = 60
    rc, w, V = _heig(np.zeros((m, m), np.complex128, order="F"))
    assert rc == 0 and not w.any()
    assert np.abs(V.conj().T @ V - np.eye(m)).max() <= 2 * m * 2.3e-16
    d = np.random.default_rng(1).permutation(np.arange(m, dtype=float))
    rc, w, V = _heig(np.asfortranarray(np.diag(d).astype(np.complex128)))
    assert rc == 0 and np.abs(w - np.arange(m)).max() <= 2 * m * 2.3e-16 * m
    A = _matrix("generic", m, np.random.default_rng(2))
    A[7, 3] = np.nan
    rc, _, _ = _heig(A)
    assert rc != 0

"""FP64 H.X on columns that fall by many orders of magnitude inside a tile:
every point is as accurate as its own stencil, on coarse meshes too."""
import ctypes as C

import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from conftest import random_fields
from nuclearcgm_gb300 import abi
from oracle import oracle

pytestmark = pytest.mark.gpu


def _reach(v, n):
    """Largest |v| over the stencil of every point; v: [cols][k][j][i]."""
    out = v.copy()
    for ax in (1, 2, 3):
        for d in (1, 2):
            lo, hi = [slice(None)] * 4, [slice(None)] * 4
            lo[ax], hi[ax] = slice(0, n - d), slice(d, n)
            out[tuple(lo)] = np.maximum(out[tuple(lo)], v[tuple(hi)])
            out[tuple(hi)] = np.maximum(out[tuple(hi)], v[tuple(lo)])
    return out


# exp(-kappa r): coarse and fine meshes, tails of 5e-2 down to 1e-14 per tile;
# and a column that falls from its first to its last plane
@pytest.mark.parametrize("n,h,kappa", [(16, 2.0, 1.0), (16, 1.5, 1.0),
                                       (20, 1.5, 1.5), (17, 0.8, 0.9),
                                       (36, 0.55, 1.5), (24, 0.8, None)])
def test_every_point_keeps_its_digits(n, h, kappa):
    f, gradf, U, W, UC = random_fields(n, 11, coulomb=True)
    a = 0.5 * (n - 1) * h
    H = ng.Hamiltonian(ng.Context(ng.Grid(n, a), 4), abi.NEUTRON)
    H.set_fields(f, gradf, U, W, UC)
    ax = (np.arange(n) - 0.5 * (n - 1)) * h
    z, y, x = np.meshgrid(ax, ax, ax, indexing="ij")
    if kappa is None:
        fall = 10.0 ** (-60.0 * (z - ax[0]) / (ax[-1] - ax[0]))
    else:
        fall = np.exp(-kappa * np.sqrt(x * x + y * y + z * z))
    rng = np.random.default_rng(5)
    X = np.stack([np.outer(fall.reshape(-1), rng.normal(size=2) +
                           1j * rng.normal(size=2)).reshape(-1)
                  for _ in range(3)], axis=1)
    Y = H.apply(np.asfortranarray(X))
    ref = oracle.Hamiltonian.skyrme(n, a, f, gradf, U, W, UC).apply(
        np.asfortranarray(X))
    err = np.abs(Y - ref).T.reshape(3, n, n, n, 2).max(axis=-1)
    big = np.abs(X).T.reshape(3, n, n, n, 2).max(axis=-1)
    # the row's sum of |coefficients| bounds |Y| / max|X|; the oracle's FP64
    # sums of up to 25 products are the larger part of the difference
    row = (np.abs(U + UC) + (7.5 + 8.5) * f / h ** 2 +
           (np.abs(gradf).reshape(3, -1).sum(0) +
            2 * np.abs(W).reshape(3, -1).sum(0)) * 18 / (12 * h))
    assert (err <= 25 * 2.0 ** -53 * row.reshape(n, n, n) *
            _reach(big, n)).all()


def _device(H, X, cols):
    import torch
    x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    ng._check(ng.load().ncgm_apply_h_device(
        H.ctx.h, H.species, x.data_ptr(), y.data_ptr(), cols, abi.FP64,
        C.c_double(0.0)))
    torch.cuda.synchronize()
    return y.cpu().numpy().T


@pytest.mark.parametrize("n", [12, 15, 16, 31])
def test_mirror_images_agree_to_the_bit(n):
    """r -> -r with the fields' parity, X -> -X and, in the integer form, X -> i
    X: the arithmetic has no preferred side (a symmetric nucleus stays where it
    is)."""
    rng = np.random.default_rng(n)
    ns, cols = n ** 3, 3
    f, gradf, U, W, UC = random_fields(n, 3, coulomb=True)
    back = slice(None, None, -1)
    H, M = (ng.Hamiltonian(ng.Context(ng.Grid(n, 0.3 * (n - 1)), cols),
                           abi.NEUTRON) for _ in range(2))
    H.set_fields(f, gradf, U, W, UC)
    M.set_fields(*(np.ascontiguousarray(v) for v in (
        f[back], -gradf.reshape(3, ns)[:, back].reshape(-1), U[back],
        -W.reshape(3, ns)[:, back].reshape(-1), UC[back])))
    r2 = np.sum(((np.indices((n, n, n)) - 0.5 * (n - 1)) * 0.6) ** 2, axis=0)
    X = (rng.normal(size=(ns, 2, cols)) + 1j * rng.normal(
        size=(ns, 2, cols))) * np.exp(-0.2 * r2).reshape(-1)[:, None, None]

    def apply(h, x):
        return _device(h, x.reshape(2 * ns, cols), cols).reshape(x.shape)

    Y = apply(H, X)
    assert np.array_equal(apply(M, X[back]), Y[back])
    assert np.array_equal(apply(H, -X), -Y)
    assert n < 15 or np.array_equal(apply(H, 1j * X), 1j * Y)

"""Edges of the lattice kernels' work splits: the density kernel at lattices
where every point lies in a lower-order boundary rule, with device, misaligned
device and host columns; the Coulomb solver's axis transforms on both sides of
their switch of lines per block and at a ragged last block."""
import ctypes as C

import numpy as np
import pytest
import torch

import nuclearcgm_gb300 as ng
from conftest import random_block
from oracle import oracle

pytestmark = pytest.mark.gpu


def _densities(ctx, ptr, cols):
    ns = ctx.grid.n ** 3
    out = [np.zeros(ns), np.zeros(ns), np.zeros(9 * ns), np.zeros(ns)]
    ng._check(ng.load().ncgm_densities(ctx.h, ptr, cols,
                                       *[o.ctypes.data for o in out]))
    return out


@pytest.mark.parametrize("n,cols", [(5, 1), (6, 3), (7, 2), (9, 1), (37, 2)])
def test_density_edges(n, cols):
    """Sums of fewer than 400 products of values of one size, each a few
    roundings of 1.1e-16 off: 1e-12 of the largest value leaves room for both
    sides. Where the columns lie makes no difference to a bit."""
    a = 0.5 * (n - 1) * 0.8
    ctx = ng.Context(ng.Grid(n, a), 8)
    Phi = np.asfortranarray(random_block(2 * n ** 3, cols, n) * 0.1)
    got = _densities(ctx, Phi.ctypes.data, cols)
    for g, ref in zip(got, (oracle.density(n, a, Phi),
                            oracle.kinetic_density(n, a, Phi),
                            oracle.so_density(n, a, Phi).T.ravel(),
                            oracle.divj(n, a, Phi))):
        assert np.abs(g - ref).max() <= 1e-12 * max(np.abs(ref).max(), 1e-30)
    flat = torch.from_numpy(Phi.ravel(order="K").view(np.float64).copy())
    dev = torch.zeros(flat.numel() + 1, dtype=torch.float64, device="cuda")
    for shift in (0, 1):  # 16-byte and 8-byte aligned
        dev[shift:shift + flat.numel()] = flat.cuda()
        torch.cuda.synchronize()
        again = _densities(ctx, dev.data_ptr() + 8 * shift, cols)
        for g, x in zip(got, again):
            assert np.array_equal(g, x)


def test_density_nan_derivative_is_zero():
    """A derivative with a NaN part counts as zero: one NaN in a column leaves
    tau finite away from that point's neighbours and at them."""
    n, a = 12, 5.0
    ctx = ng.Context(ng.Grid(n, a), 2)
    Phi = np.asfortranarray(random_block(2 * n ** 3, 1, 3) * 0.1)
    at = 6 + n * (6 + n * 6)
    Phi[2 * at, 0] = complex(np.nan, 0.0)
    rho, tau, J9, divj = _densities(ctx, Phi.ctypes.data, 1)
    assert np.isnan(rho[at]) and np.isfinite(np.delete(rho, at)).all()
    assert np.isfinite(tau).all()
    near = np.delete(np.arange(n ** 3), at)
    assert np.isfinite(divj[near]).all()
    assert np.isfinite(J9.reshape(9, -1)[:, near]).all()


@pytest.mark.parametrize("n", [9, 11, 34, 35, 37])
def test_poisson_edges(n):
    """The direct potential against the oracle's, at the tolerance of the
    solver's own parity test."""
    a = 0.5 * (n - 1) * 0.7
    xs = -a + np.arange(n) * 2 * a / (n - 1)
    z, y, x = np.meshgrid(xs, xs, xs, indexing="ij")
    rho = np.exp(-((x - 0.3) ** 2 + (y + 0.2) ** 2 + 1.2 * z ** 2) / 2.2).ravel()
    Z = 8
    rho *= Z / oracle.integral(n, a, rho)
    ctx = ng.Context(ng.Grid(n, a), 2)
    U = np.zeros(n ** 3)
    its = C.c_int(0)
    ng._check(ng.load().ncgm_poisson(ctx.h, rho.ctypes.data, Z, None,
                                     U.ctypes.data, None, C.byref(its)))
    ref, _ = oracle.poisson(n, a, rho, Z)
    assert np.abs(U - ref).max() <= 1e-9 * np.abs(ref).max()

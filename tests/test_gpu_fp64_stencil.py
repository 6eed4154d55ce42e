"""The FP64 Hamiltonian product (integer form, k_stencil64.cu) at the edges of
its tiles and of its number format, against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from conftest import random_block, random_fields
from nuclearcgm_gb300 import abi
from oracle import oracle

pytestmark = pytest.mark.gpu


def _pair(n, seed=1, cols=70):
    f, gradf, U, W, UC = random_fields(n, seed, coulomb=True)
    a = 0.5 * (n - 1) * 0.8
    H = ng.Hamiltonian(ng.Context(ng.Grid(n, a), cols), abi.NEUTRON)
    H.set_fields(f, gradf, U, W, UC)
    return H, oracle.Hamiltonian.skyrme(n, a, f, gradf, U, W, UC)


def _shifted(H, X, shift):
    import torch
    x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    ng._check(ng.load().ncgm_apply_h_device(
        H.ctx.h, H.species, x.data_ptr(), y.data_ptr(), X.shape[1], abi.FP64,
        C.c_double(shift)))
    torch.cuda.synchronize()
    return y.cpu().numpy().T


# the FP64 kernel of small lattices, then ragged and even tilings of the
# integer form; more than 64 columns split a block's column group. Errors are 2^-53 of the largest
# |H| |x| a row can form, which is below 4 max|Y| for random blocks.
@pytest.mark.parametrize("n,cols", [(4, 1), (9, 2), (14, 5), (15, 1), (15, 70),
                                    (16, 65), (17, 3), (23, 4), (31, 2)])
def test_matches_oracle(n, cols):
    H, R = _pair(n)
    X = random_block(2 * n ** 3, cols, n)
    ref = R.apply(X)
    assert np.abs(H.apply(X) - ref).max() <= 1e-14 * np.abs(ref).max()


def test_scale_is_local():
    """A column that falls by 10^-60 over the lattice keeps FP64's relative
    accuracy far from its maximum: every tile has its own scale."""
    n = 24
    H, R = _pair(n)
    x = np.arange(n)
    fall = np.repeat(10.0 ** (-60.0 * x / n)[:, None] *
                     np.ones((1, n * n)), 2, axis=1).reshape(-1)
    X = np.asfortranarray(random_block(2 * n ** 3, 2, 3) * fall[:, None])
    ref, Y = R.apply(X), H.apply(X)
    plane = np.abs(ref).reshape(n, -1).max(axis=1)
    err = np.abs(Y - ref).reshape(n, -1).max(axis=1)
    # a tile spans up to 9 + 4 planes of a factor 316 each at the most; the
    # integers hold 2^-58 of its largest value
    assert (err <= 1e-14 * plane + 2.0 ** -50 * np.array(
        [plane[max(0, k - 12):k + 1].max() for k in range(n)])).all()


@pytest.mark.parametrize("scale", [0.0, 1e-290, 1e-200, 1e200, 1e300])
def test_magnitudes(scale):
    n = 16
    H, R = _pair(n)
    X = random_block(2 * n ** 3, 3, 5)
    X[:, 1] *= scale
    ref = R.apply(X)
    Y = H.apply(X)
    for c in range(3):
        m = np.abs(ref[:, c]).max()
        assert np.abs(Y[:, c] - ref[:, c]).max() <= 1e-14 * m + 5e-323


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_values_stay_local(value):
    n = 20
    H, R = _pair(n)
    X = random_block(2 * n ** 3, 3, 6)
    clean = H.apply(X)
    p = 2 * (7 + n * (9 + n * 11))
    X[p, 1] = value
    Y, ref = H.apply(X), R.apply(X)
    assert np.array_equal(np.isfinite(Y), np.isfinite(ref))
    good = np.isfinite(ref)
    assert np.abs(Y[good] - clean[good]).max() <= 1e-14 * np.abs(clean).max()


@pytest.mark.parametrize("shift", [47.3, -300.0, 1e9])
def test_shift(shift):
    """Shifts inside and beyond the coefficients' format."""
    n = 17
    H, R = _pair(n)
    X = random_block(2 * n ** 3, 4, 7)
    ref = R.apply(X) + shift * X
    Y = _shifted(H, X, shift)
    assert np.abs(Y - ref).max() <= 1e-14 * np.abs(ref).max()

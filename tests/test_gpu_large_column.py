"""A start column whose norm overflows: its pivot of the orthonormalisation is
infinite, what it divides becomes zero, and the call goes on without it."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi, config, workloads

pytestmark = pytest.mark.gpu


def test_overflowing_column_is_dropped():
    n, nev = 10, 5
    a, f, gradf, U, W = workloads.fields(n, 0.9)
    H = ng.Hamiltonian(ng.Context(ng.Grid(n, a), 32), abi.NEUTRON)
    H.set_fields(f, gradf.T, U, W.T)
    X = workloads.orthonormal_block(2 * n ** 3, nev, seed=5)
    X[:, 1] *= 1e170
    prm = config._gcg(config.HF_GCG)
    Xo, lam, st = H.gcg(np.asfortranarray(X), nev, None, prm)
    assert np.isfinite(lam).all() and np.isfinite(Xo).all()

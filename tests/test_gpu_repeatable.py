"""The same call on the same input gives the same bits in every precision form,
also with search spaces wider than one warp's rows (the triangular factor's
rows then go to several warps)."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi, config, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32, abi.FP32_TC])
def test_gcg_repeats_to_the_bit(precision):
    n, nev = 16, 20
    a, f, gradf, U, W = workloads.fields(n, 0.8)
    H = ng.Hamiltonian(ng.Context(ng.Grid(n, a), 4 * nev), abi.NEUTRON)
    H.set_fields(f, gradf.T, U, W.T)
    X = workloads.orthonormal_block(2 * n ** 3, nev, seed=3)
    P = workloads.orthonormal_block(2 * n ** 3, nev, seed=4)
    prm = config._gcg(config.HF_GCG, precision)
    first = None
    for _ in range(40 if precision == abi.FP64 else 120):
        Xo, lam, _ = H.gcg(X, nev, P, prm)
        if first is None:
            first = Xo.copy(), lam.copy()
        assert np.array_equal(lam, first[1]) and np.array_equal(Xo, first[0])


def test_hf_run_repeats_to_the_bit():
    """Both species' eigenproblems at once, 20 orbitals and 20 directions each
    (60 columns)."""
    cfg = config.from_input({
        "functional": "SLy4", "nucleus": {"A": 40, "Z": 20},
        "box": {"boxSize": 16.0, "axisMeshPoints": 24},
        "maxIterations": 12, "energyTol": 0.0})
    cfg.hf_gcg.precision = abi.FP32
    runs = [ng.hf_run(cfg) for _ in range(6)]
    for res, out in runs[1:]:
        assert res.E_int == runs[0][0].E_int
        assert np.array_equal(out["rho_n"], runs[0][1]["rho_n"])

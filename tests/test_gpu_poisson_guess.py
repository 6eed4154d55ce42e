"""A Coulomb solve that fails leaves the potential that serves as the next
guess as it was: a self-consistent state recovers with its next update."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi, config
from test_gpu_state import BOX, N_LAT, _orbitals, _rel

pytestmark = pytest.mark.gpu


def test_update_after_a_failed_solve():
    # no mixing: the densities are those of the last update alone
    cfg = config.from_input({
        "functional": "SLy4", "nucleus": {"A": 16, "Z": 8},
        "box": {"boxSize": BOX, "axisMeshPoints": N_LAT}, "densityMix": 1.0,
        "maxIterations": 1, "energyTol": 0.0})
    n = (_orbitals(N_LAT, BOX, 8, 1), np.linspace(-40.0, -5.0, 8))
    p = (_orbitals(N_LAT, BOX, 8, 2), np.linspace(-35.0, -2.0, 8))
    # a charge whose residual norm overflows
    huge = (p[0] * 1e100, p[1])
    one, two = ng.IterationData(cfg), ng.IterationData(cfg)
    for st in (one, two):
        st.update_quantities(n, p, 0, abi.UPDATE_NORMALIZE)
    with pytest.raises(RuntimeError):
        one.update_quantities(n, huge, 1, 0)
    q = (_orbitals(N_LAT, BOX, 8, 3), p[1])
    for st in (one, two):
        st.update_quantities(n, q, 2, abi.UPDATE_NORMALIZE)
    for a, b in zip(one.fields(abi.PROTON), two.fields(abi.PROTON)):
        assert _rel(a, b) < 1e-9
    one.close()
    two.close()

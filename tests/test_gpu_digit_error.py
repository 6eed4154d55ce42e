"""A tensor-core kernel whose bounded wait ran out is reported by its own
context and by no other one: several contexts run digit products at once (the
two species of a self-consistent run, batched runs)."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi

pytestmark = pytest.mark.gpu

TIMEOUT = 5
N = 15


def _gram(ctx):
    A = np.asfortranarray(np.random.default_rng(1).normal(
        size=(2 * N ** 3, 6)) + 0j)
    G = np.zeros((6, 6), complex, order="F")
    return ng.load().ncgm_gram(ctx.h, A.ctypes.data, 6, A.ctypes.data, 6,
                               G.ctypes.data, abi.FP64)


def _vc(ctx):
    V = np.asfortranarray(np.random.default_rng(2).normal(
        size=(2 * N ** 3, 40)) + 0j)
    Cm = np.eye(40, dtype=complex, order="F")
    Y = np.zeros_like(V)
    return ng.load().ncgm_vc(ctx.h, V.ctypes.data, 40, Cm.ctypes.data, 40,
                             Y.ctypes.data, abi.FP64)


@pytest.mark.parametrize("call", [_gram, _vc])
def test_own_context_reports_it(call):
    one, two = (ng.Context(ng.Grid(N, 4.2), 4) for _ in range(2))
    for c in (one, two):
        assert call(c) == 0
    ng._check(ng.load().ncgm_set_digit_error(one.h))
    assert call(two) == 0
    assert call(one) == TIMEOUT
    assert call(one) == 0  # reported once
    assert call(two) == 0

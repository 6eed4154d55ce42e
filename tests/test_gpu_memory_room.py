"""The digit images of the FP64 block products are scratch of a faster form:
they are taken only while as much memory again stays free, after everything
that the call cannot do without, and the plain kernels give the same result."""
import numpy as np
import pytest

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi, config, workloads

pytestmark = pytest.mark.gpu


def _gcg(n, nev, X, P):
    a, f, gradf, U, W = workloads.fields(n, 0.8)
    ctx = ng.Context(ng.Grid(n, a), 3 * nev + P.shape[1])
    H = ng.Hamiltonian(ctx, abi.NEUTRON).set_fields(f, gradf.T, U, W.T)
    _, lam, _ = H.gcg(X, nev, P, config._gcg(config.HF_GCG))
    return ctx, lam


def test_images_leave_room():
    import torch
    n, nev = 24, 20
    N, v = 2 * n ** 3, 4 * nev
    X = workloads.orthonormal_block(N, nev, seed=3)
    P = workloads.orthonormal_block(N, nev, seed=4)
    ctx, free_run = _gcg(n, nev, X, P)
    ctx.close()
    # blocks of the search space, of the levels and of the corrections, the
    # plain products' partials, the staged arguments
    base = 16 * (4 * N * v + (5 + 7) * N * nev + 3 * N * nev +
                 (256 + 8) * v * v)
    images = 64 * N * v
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    room = base + (64 << 20) + int(1.3 * images)
    fill = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        ctx, lam = _gcg(n, nev, X, P)
        left = torch.cuda.mem_get_info()[0]
        ctx.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    assert left >= images
    assert np.allclose(lam, free_run, rtol=1e-6)

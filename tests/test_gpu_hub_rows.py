"""Rows with tens of thousands of entries: a hub joined to all other cells.

The hub's lower-side count takes 16 bits (above 32,767 the sign bit of the
word that holds it).  Everything that walks over a row in two parts
is bit-identical to the oracle (same entry order and roundings, so the
tolerance is zero); Krylov solutions, whose dot products are summed in another
order, agree to 1e-10.
"""
import time

import numpy as np
import pytest

from oracle_lib import OracleAmg
from unap_gb300 import capi
from unap_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def hub_system(below, above, symm, seed):
    """Cell `below` joined to `below` cells before and `above` cells after it."""
    rng = np.random.default_rng(seed)
    n = below + above + 1
    l = np.concatenate([np.arange(below), np.full(above, below)]).astype(np.int32)
    u = np.concatenate([np.full(below, below), np.arange(below + 1, n)]).astype(np.int32)
    upper = -rng.random(n - 1) - 0.1
    lower = upper if symm else -rng.random(n - 1) - 0.1
    diag = W._fast_row_abs_sum(n, l, u, upper, lower) + 1.0
    return W.LduSystem(n, l, u, None if symm else lower, diag, upper, rng.standard_normal(n))


HUBS = [(40_000, 0), (35_000, 5_000), (33_000, 32_535)]


@pytest.mark.parametrize("below,above", HUBS)
def test_sweeps_and_preconditioners(cuda, orc, below, above):
    torch = cuda
    s = hub_system(below, above, False, 1)
    A = capi.DeviceMatrix(s)
    x0 = np.random.default_rng(2).standard_normal(s.n)
    b = torch.tensor(s.b, device="cuda")
    for backward in (False, True):
        for sweeps in (1, 3):
            x = torch.tensor(x0, device="cuda")
            A.gauss_seidel(x, b, sweeps, backward=backward)
            assert np.array_equal(x.cpu().numpy(), orc.gs(s, x0, s.b, sweeps, backward=backward))
    w = torch.zeros(s.n, dtype=torch.float64, device="cuda")
    for t in (2, 3):
        A.precondition(t, torch.tensor(x0, device="cuda"), w)
        assert np.array_equal(w.cpu().numpy(), orc.precond(t, s, x0)[0]), t
    A.close()


@pytest.mark.parametrize("shape", [None, (256, 1), (256, 8)])
@pytest.mark.parametrize("method,precond", [(0, 2), (1, 3)])
def test_krylov(cuda, orc, shape, method, precond):
    """Per-step launches and whole-solve launches of one CTA and of a cluster."""
    torch = cuda
    s = hub_system(35_000, 5_000, method == 0, 3)
    ref, st_ref = (orc.pcg if method == 0 else orc.pbicgstab)(s, precond, s.b, rel_tol=1e-11)
    old = capi.set_team_solve_cells(1 << 20 if shape else 0)
    if shape:
        capi.force_team_shape(*shape)
    try:
        A = capi.DeviceMatrix(s)
        x = torch.zeros(s.n, dtype=torch.float64, device="cuda")
        st = A.krylov_solve(method, precond, x, torch.tensor(s.b, device="cuda"), rel_tol=1e-11)
        A.close()
    finally:
        capi.set_team_solve_cells(old)
        capi.force_team_shape(0)
    assert st["converged"] and abs(st["nIterations"] - st_ref["n_iter"]) <= 1
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("packed", [0, 1, 2])
def test_vcycle_sweeps(cuda, orc, precision, packed):
    """A hierarchy built by host loops; its sweeps in one launch and as
    launches per wavefront, with SELL-32 and with row-packed rows."""
    torch = cuda
    s = hub_system(40_000, 0, True, 4)
    r = np.random.default_rng(5).standard_normal(s.n)
    old_setup, old_packed = capi.set_device_setup(-1), capi.set_packed_sweeps(packed)
    try:
        A = capi.DeviceMatrix(s)
        G = capi.DeviceAmg(A, n_coarsest=10, precision=precision)
        O = OracleAmg(orc, s, n_coarsest=10, precision=precision)
        assert G.info()["cells"] == O.level_sizes()
        z = torch.zeros(s.n, dtype=torch.float64, device="cuda")
        G.vcycle(torch.tensor(r, device="cuda"), z)
        assert np.array_equal(z.cpu().numpy(), O.vcycle(r))
        G.close()
        O.close()
        A.close()
    finally:
        capi.set_device_setup(old_setup)
        capi.set_packed_sweeps(old_packed)


@pytest.mark.parametrize("leaves", [2047, 2048, 2049, 40_000])
def test_hierarchy_with_a_large_aggregate(cuda, orc, leaves):
    """All cells around the hub join its aggregate.  Up to the longest list the
    setup kernels sort (2,048) and beyond it, the transfers are the host's and
    the setup takes no longer than for any system of the size."""
    torch = cuda
    s = hub_system(leaves, 0, True, 6)
    r = np.random.default_rng(7).standard_normal(s.n)
    old = capi.set_device_setup(1000)
    try:
        A = capi.DeviceMatrix(s)
        t0 = time.perf_counter()
        G = capi.DeviceAmg(A, n_coarsest=10, precision=0)
        seconds = time.perf_counter() - t0
    finally:
        capi.set_device_setup(old)
    O = OracleAmg(orc, s, n_coarsest=10, precision=0)
    assert G.info()["cells"] == O.level_sizes()
    z = torch.zeros(s.n, dtype=torch.float64, device="cuda")
    G.vcycle(torch.tensor(r, device="cuda"), z)
    assert np.array_equal(z.cpu().numpy(), O.vcycle(r))
    assert seconds < 5.0
    G.close()
    O.close()
    A.close()

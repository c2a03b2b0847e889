"""Products over large levels, where a warp walks over several slices, and in the caller's order.

The products are bit-identical to the oracle's (the same entry order and
roundings, tolerance zero) at the sizes where the walk can go wrong: the last
block of 256 rows and the last slice partly filled, rows longer than the eight
entries held in registers, products of -0, rows without entries.  The dot
products sum the same terms as the oracle's in another order: at most n eps =
6e-11 of the sum of their magnitudes, so three iterations of a
well-conditioned solve agree to 1e-9.
"""
import numpy as np
import pytest

from test_gpu_flow import random_system
from unap_gb300 import capi

pytestmark = pytest.mark.gpu

LIMIT = 1 << 19  # rows from which FP64 levels are walked


@pytest.mark.parametrize("n,per_row", [(LIMIT, 2.2), (LIMIT + 1, 3.0), (LIMIT + 31 * 256 + 45, 0.3),
                                       (LIMIT - 1, 2.2)])
@pytest.mark.parametrize("symm", [True, False])
def test_products_and_dots(cuda, orc, n, per_row, symm):
    torch = cuda
    s = random_system(n, int(per_row * n), n % 97, symm=symm, near=9000)
    A = capi.DeviceMatrix(s)
    x = np.random.default_rng(n).standard_normal(n)
    x[::5] = -0.0
    y = torch.empty(n, dtype=torch.float64, device="cuda")
    A.spmv(torch.tensor(x, device="cuda"), y)
    want = orc.spmv(s, x)
    assert np.array_equal(y.cpu().numpy().view(np.int64), want.view(np.int64))
    z = torch.zeros(n, dtype=torch.float64, device="cuda")
    A.krylov_solve(0 if symm else 1, 1, z, torch.tensor(s.b, device="cuda"),
                   rel_tol=0.0, max_iter=3)
    ref = (orc.pcg if symm else orc.pbicgstab)(s, 1, s.b, rel_tol=0.0, max_iter=3)
    xr, _ = ref
    assert np.abs(z.cpu().numpy() - xr).max() <= 1e-9 * np.abs(xr).max()
    A.close()


@pytest.mark.parametrize("n", [1, 33, 5000, 40_000, LIMIT - 1, LIMIT])
@pytest.mark.parametrize("shift", [None, 0, 1, 32])
def test_products_in_the_callers_order(cuda, orc, n, shift):
    """y apart from x, x itself, or x moved by some entries."""
    torch = cuda
    s = random_system(n, int(2.2 * n) if n > 1 else 0, n % 89, near=min(n, 9000) if n > 1 else None)
    A = capi.DeviceMatrix(s)
    x = np.random.default_rng(n).standard_normal(n)
    buf = torch.zeros(2 * n + 32, dtype=torch.float64, device="cuda")
    buf[:n] = torch.tensor(x)
    at = n if shift is None else min(shift, n)
    A.spmv(buf[:n], buf[at:at + n])
    assert np.array_equal(buf[at:at + n].cpu().numpy(), orc.spmv(s, x))
    A.close()


@pytest.mark.parametrize("exponent", [0, -126, -128])
def test_fp32_cycles_near_the_smallest_numbers(cuda, exponent):
    """FP32 results widened to FP64: normal and subnormal numbers, zeros,
    infinities.  Scaling the right-hand side by a power of two scales the
    result but for roundings to multiples of 2^-149: some 10^4 of them, of
    1.4e-45 each, against results of 1e-39 and more."""
    torch = cuda
    s = random_system(4000, 9000, 5, symm=True, near=300)
    A = capi.DeviceMatrix(s)
    G = capi.DeviceAmg(A, precision=1, n_coarsest=100)
    z = torch.empty(s.n, dtype=torch.float64, device="cuda")

    def cycle(b):
        G.vcycle(torch.tensor(b, device="cuda"), z)
        return z.cpu().numpy().copy()

    want = cycle(s.b) * 2.0 ** exponent
    got = cycle(s.b * 2.0 ** exponent)
    assert np.array_equal(got, got.astype(np.float32).astype(np.float64))
    if exponent == 0:
        assert np.array_equal(got, want)
    assert np.abs(got - want).max() <= 1e4 * 2.0 ** -149 or exponent == 0
    assert np.array_equal(cycle(0.0 * s.b), np.zeros(s.n))
    b = s.b.copy()
    b[7] = np.inf
    assert not np.isfinite(cycle(b)).all()
    G.close()
    A.close()


@pytest.mark.parametrize("leaves", [255, 256, 257, 3000])
@pytest.mark.parametrize("entries", [8, 20])
def test_products_with_a_long_row(cuda, orc, leaves, entries):
    """A row on each side of the longest one whose columns are looked up, in
    systems of short and of longer rows; more than 2^20 entries are left to
    the copying form too."""
    torch = cuda
    n = 60_000
    g = random_system(n, n * entries // 2, 7, near=2000)
    key = np.concatenate([g.lower_addr.astype(np.int64) * (n + 1) + g.upper_addr,
                          np.arange(leaves).astype(np.int64) * (n + 1) + n])
    order = np.argsort(key)
    rng = np.random.default_rng(leaves)
    s = type(g)(n + 1, (key[order] // (n + 1)).astype(np.int32),
                (key[order] % (n + 1)).astype(np.int32), rng.standard_normal(key.size),
                rng.standard_normal(n + 1), rng.standard_normal(key.size),
                rng.standard_normal(n + 1))
    A = capi.DeviceMatrix(s)
    x = rng.standard_normal(s.n)
    y = torch.empty(s.n, dtype=torch.float64, device="cuda")
    A.spmv(torch.tensor(x, device="cuda"), y)
    assert np.array_equal(y.cpu().numpy(), orc.spmv(s, x))
    A.close()

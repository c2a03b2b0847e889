"""Gauss-Seidel sweeps and DIC/DILU in one launch: rows wait for their neighbours by value.

Bit-identical to the oracle's sweeps (the same entry order and roundings, so
the tolerance is zero) at the sizes where the launch can go wrong: single
rows, wavefronts of one row, tasks cut at slice and wavefront boundaries, rows
longer than a chunk, every lane count of the size rule, more sweeps than one
launch takes, and NaNs with the bit pattern that marks a value still missing.
"""
import numpy as np
import pytest

from unap_gb300 import capi
from unap_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def random_system(n, faces, seed, symm=False, near=None):
    """About `faces` random faces (distinct pairs, at most `near` cells apart),
    owner-sorted, diagonally dominant."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, n, faces)
    d = rng.integers(1, (near or n), faces)
    b = a + d
    ok = b < n
    key = np.unique(a[ok].astype(np.int64) * n + b[ok])
    l, u = (key // n).astype(np.int32), (key % n).astype(np.int32)
    upper = rng.standard_normal(l.size)
    lower = upper if symm else rng.standard_normal(l.size)
    diag = W._fast_row_abs_sum(n, l, u, upper, lower) + 1.0
    return W.LduSystem(n, l, u, None if symm else lower, diag, upper, rng.standard_normal(n))


CASES = {
    "one_cell": lambda: random_system(1, 0, 1),
    "no_faces_33": lambda: random_system(33, 0, 2),
    "chain_70": lambda: W.laplace(70, 1, 1, seed=3),           # 70 wavefronts of one row
    "plane_31x33": lambda: W.laplace(31, 33, 1, seed=4),       # wavefronts of 1 to 31 rows
    "grid_7pt": lambda: W.convdiff(17, 13, 11, seed=5),
    "rows_of_45": lambda: random_system(300, 9000, 6),         # longer than any chunk
    "rows_of_20": lambda: random_system(2500, 25000, 7, symm=True),
    "wide_4_lanes": lambda: random_system(160_000, 900_000, 8, near=4000),
    "wide_1_lane": lambda: random_system(310_000, 1_700_000, 9, near=9000),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("backward", [False, True])
def test_sweeps_bit_exact(cuda, orc, name, backward):
    torch = cuda
    s = CASES[name]()
    A = capi.DeviceMatrix(s)
    x0 = np.random.default_rng(s.n).standard_normal(s.n)
    b = torch.tensor(s.b, device="cuda")
    for sweeps in ((1, 2) if s.n > 100_000 else (1, 4, 5, 9)):
        x = torch.tensor(x0, device="cuda")
        A.gauss_seidel(x, b, sweeps, backward=backward)
        assert np.array_equal(x.cpu().numpy(), orc.gs(s, x0, s.b, sweeps, backward=backward)), sweeps
    A.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_preconditioners_bit_exact(cuda, orc, name):
    torch = cuda
    s = CASES[name]()
    A = capi.DeviceMatrix(s)
    r = np.random.default_rng(s.n + 1).standard_normal(s.n)
    for t in (2, 3):
        w = torch.zeros(s.n, dtype=torch.float64, device="cuda")
        A.precondition(t, torch.tensor(r, device="cuda"), w)
        assert np.array_equal(w.cpu().numpy(), orc.precond(t, s, r)[0], equal_nan=True), t
    A.close()


@pytest.mark.parametrize("pattern", [0xFFFFFFFFFFFFFFFF, 0x7FF8000000000000, 0x7FF0000000000000])
def test_nan_and_inf_inputs(cuda, orc, pattern):
    """A NaN that looks like a missing value, another NaN and an infinity
    spread as in the oracle, and no wait runs out on them."""
    torch = cuda
    s = W.laplace(9, 8, 7, seed=1, permute=True)
    bad = np.array([pattern], dtype=np.uint64).view(np.float64)[0]
    A = capi.DeviceMatrix(s)
    for where in ("b", "x"):
        x0 = np.random.default_rng(2).standard_normal(s.n)
        b = s.b.copy()
        (b if where == "b" else x0)[s.n // 2] = bad
        x = torch.tensor(x0, device="cuda")
        A.gauss_seidel(x, torch.tensor(b, device="cuda"), 2)
        assert np.array_equal(x.cpu().numpy(), orc.gs(s, x0, b, 2), equal_nan=True)
        if where == "b":
            A.precondition(2, torch.tensor(b, device="cuda"), x)
            assert np.array_equal(x.cpu().numpy(), orc.precond(2, s, b)[0], equal_nan=True)
    A.close()


@pytest.mark.parametrize("degree", [1, 3, 4])
@pytest.mark.parametrize("precision", [0, 1])
def test_chebyshev_tail_long_rows(cuda, precision, degree):
    """The Chebyshev tail from level 1 on a hierarchy whose rows are longer
    than the entries a task holds at once: the bits of a launch per step."""
    torch = cuda
    s = random_system(3000, 60000, 11, symm=True)
    s.upper = s.upper * 0 - np.abs(s.upper)
    s.diag = W._fast_row_abs_sum(s.n, s.lower_addr, s.upper_addr, s.upper, s.upper) + 0.1
    A = capi.DeviceMatrix(s)
    r = torch.tensor(np.random.default_rng(3).standard_normal(s.n), device="cuda")
    out = []
    for rows in (0, 1 << 30):
        old = capi.set_cheby_tail_rows(rows)
        try:
            G = capi.DeviceAmg(A, n_coarsest=70, precision=precision, smoother=1,
                               cheby_degree=degree)
        finally:
            capi.set_cheby_tail_rows(old)
        z = torch.zeros_like(r)
        G.vcycle(r, z)
        out.append(z.cpu().numpy())
        G.close()
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
    A.close()


def test_matrix_keeps_one_vector_a_sweep(cuda):
    """Four sweeps leave four vectors (and the call's two) with the matrix."""
    torch = cuda
    s = W.laplace(160, 160, 80, seed=1)
    A = capi.DeviceMatrix(s)
    b = torch.tensor(s.b, device="cuda")
    x = torch.zeros_like(b)
    A.spmv(b, x)  # the call's two vectors
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    A.gauss_seidel(x, b, 4)
    free1, _ = torch.cuda.mem_get_info()
    assert free0 - free1 <= 4 * 8 * s.n + (4 << 20)
    A.close()

"""The coarsest level's kernels at the edges of their ranges: factors of 1 to
64 unknowns (and 65, the general kernel) after a resetup against the setup's
host factors bit for bit, the l1 diagonals of short, long and empty-tailed
rows (a thread, or a warp per 4 or 16 rows), and cycles through the explicit inverse against the oracle."""

import numpy as np
import pytest
import scipy.sparse as sp

import draugr
import oracle
from draugr import problems

pytestmark = pytest.mark.gpu


def dense_system(n, seed):
    """Random dense couplings, so that the factorisation pivots."""
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1, 1, (n, n)) + np.diag(rng.uniform(0, 1, n))
    return sp.csr_matrix(A)


def zero_diagonal_system(n, seed):
    """Diagonally dominant rows dealt in cyclic order: every diagonal entry is
    exactly zero, and the first n - 1 columns need an interchange."""
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1, 1, (n, n)) + 2 * n * np.eye(n)
    A = np.roll(A, 1, axis=0)
    A[np.arange(n), np.arange(n)] = 0.0
    return sp.csr_matrix(A)


@pytest.mark.parametrize("system", [dense_system, zero_diagonal_system])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 48, 63, 64, 65, 90])
def test_factors_after_resetup(n, system):
    if n == 1:
        system = dense_system
    A = system(n, n)
    cfg = draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25), smoother=draugr.JacobiSmootherType(),
                           max_coarse_size=100)
    h = draugr.amg_setup(A, cfg)  # n <= 100: the coarsest system alone
    lu, piv = h.export(-1, "C_lu"), h.export(-1, "C_piv")
    B = A.copy()
    B.data = B.data * 0.5
    draugr.amg_resetup(h, B, cfg)
    draugr.amg_resetup(h, A, cfg)
    assert np.array_equal(h.export(-1, "C_piv"), piv)
    assert np.array_equal(h.export(-1, "C_lu"), lu)


@pytest.mark.parametrize("n", [8, 64, 65, 72])
def test_factors_of_nan_values_keep_pivots_in_range(n):
    """A resetup with NaN coefficients leaves pivots that the substitutions
    can index with, and the next resetup recovers."""
    A = dense_system(n, n)
    cfg = draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25), smoother=draugr.JacobiSmootherType(),
                           max_coarse_size=100)
    h = draugr.amg_setup(A, cfg)
    lu, piv = h.export(-1, "C_lu"), h.export(-1, "C_piv")
    B = A.copy()
    B.data = np.full_like(B.data, np.nan)
    draugr.amg_resetup(h, B, cfg)
    assert np.array_equal(h.export(-1, "C_piv"), np.arange(n))
    draugr.amg_resetup(h, A, cfg)
    assert np.array_equal(h.export(-1, "C_piv"), piv)
    assert np.array_equal(h.export(-1, "C_lu"), lu)


@pytest.mark.parametrize("A", [problems.poisson1d(1000), problems.anisotropic_27pt(11), problems.anisotropic_27pt(41),
                               sp.csr_matrix(problems.poisson1d(300) + sp.eye(300) * 0 +
                                             sp.csr_matrix((np.ones(300), (np.zeros(300, int), np.arange(300))),
                                                           shape=(300, 300)))],
                         ids=["3_per_row", "27_per_row", "27_per_row_many", "one_full_row"])
def test_l1_diagonal_after_resetup(A):
    A = sp.csr_matrix(A)
    A.sort_indices()
    cfg = draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25), smoother=draugr.L1JacobiSmootherType())
    h = draugr.amg_setup(A, cfg)
    before = [h.export(l, "invdiag") for l in range(h.nlevels)]
    draugr.amg_resetup(h, A, cfg)
    for l, d in enumerate(before):
        assert np.array_equal(h.export(l, "invdiag"), d)


@pytest.mark.parametrize("coarse", [8, 33, 64, 90])
def test_cycle_through_the_coarsest_inverse(coarse):
    A = problems.heterogeneous_diffusion_3d(20, seed=2)
    cfg = draugr.hypre_default_config(agg_trunc_factor=0.2, smoother=draugr.L1JacobiSmootherType(),
                                      max_coarse_size=coarse, seed=1)
    h = draugr.amg_setup(A, cfg)
    b = problems.rhs(A.shape[0], 4)
    x = draugr.amg_cycle(np.zeros(A.shape[0]), b, h, cfg)
    ref = oracle.OracleHierarchy(h).cycle(np.zeros(A.shape[0]), b)
    assert np.linalg.norm(x - ref) < 1e-12 * np.linalg.norm(ref)


def neumann(m, shift):
    """Heterogeneous diffusion on m^3 cells without a boundary condition,
    plus `shift` on the diagonal: nearly singular on every level."""
    kap = np.exp(1.5 * np.random.default_rng(3).standard_normal(m ** 3))
    idx = np.arange(m ** 3).reshape(m, m, m)
    r, c, v = [], [], []
    for ax in range(3):
        a, b = np.take(idx, range(m - 1), ax).ravel(), np.take(idx, range(1, m), ax).ravel()
        w = 2 / (1 / kap[a] + 1 / kap[b])
        r += [a, b]
        c += [b, a]
        v += [-w, -w]
    A = sp.csr_matrix((np.concatenate(v), (np.concatenate(r), np.concatenate(c))), shape=(m ** 3, m ** 3))
    return sp.csr_matrix(A + sp.diags(shift - np.asarray(A.sum(1)).ravel())).sorted_indices()


def pcg(A, M, b, tol, maxiter):
    x, r, p, rz = np.zeros_like(b), b.copy(), None, 0.0
    for it in range(1, maxiter + 1):
        z = M(r)
        rz, old = r @ z, rz
        p = z if p is None else z + rz / old * p
        q = A @ p
        alpha = rz / (p @ q)
        x, r = x + alpha * p, r - alpha * q
        if np.linalg.norm(r) < tol * np.linalg.norm(b):
            break
    return x, it


@pytest.mark.parametrize("shift", [1e-3, 1e-6, 1e-9])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nearly_singular_coarsest_system(shift, precision):
    """The explicit inverse where it could lose most: a coarsest system of
    33 to 64 unknowns with a condition of up to 1e11.  PCG takes as many
    iterations as with the oracle's substitutions, to the same residual."""
    A = neumann(32, shift)
    cfg = draugr.hypre_default_config(agg_trunc_factor=0.2, smoother=draugr.L1JacobiSmootherType(), seed=3,
                                      max_coarse_size=64)
    h = draugr.amg_setup(A, cfg)
    assert 33 <= int(h.level_info(-1)[0]) <= 64
    O = oracle.OracleHierarchy(h)
    b = A @ np.random.default_rng(1).uniform(-1, 1, A.shape[0])
    want, steps = pcg(A, lambda r: O.cycle(np.zeros_like(r), r), b, 1e-8, 200)
    x, it, _ = draugr.pcg(np.zeros_like(b), b, h, cfg, tol=1e-8, maxiter=200, precision=precision)
    assert abs(it - steps) <= 1
    assert np.linalg.norm(b - A @ x) < max(1.01e-8 * np.linalg.norm(b), 1.5 * np.linalg.norm(b - A @ want))

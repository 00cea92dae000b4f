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

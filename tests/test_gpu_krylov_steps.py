"""BiCGStab and FGMRES with their scalars on the device: iterates after a few
steps against NumPy with the oracle's cycle as the preconditioner (a step
enqueued past the last one must not change x), and the transposed coarsest
solve at the edges of its kernels."""

import numpy as np
import pytest

import draugr
import oracle
from draugr import problems

pytestmark = pytest.mark.gpu


def system(m=24, coarse=30):
    kappa = np.exp(0.3 * np.random.default_rng(2).standard_normal((m, m)))
    A, _ = problems.convection_diffusion_2d(kappa, 20.0, seed=3)
    cfg = draugr.hypre_default_config(agg_trunc_factor=0.2, smoother=draugr.L1JacobiSmootherType(),
                                      max_coarse_size=coarse, seed=3)
    return A, cfg, draugr.amg_setup(A, cfg), problems.rhs(m * m, 5)


def bicgstab(A, M, b, steps):
    x, r = np.zeros_like(b), b.copy()
    rh, p, v = r.copy(), np.zeros_like(b), np.zeros_like(b)
    rho = alpha = omega = 1.0
    for _ in range(steps):
        rho1 = rh @ r
        p = r + (rho1 / rho) * (alpha / omega) * (p - omega * v)
        ph = M(p)
        v = A @ ph
        alpha = rho1 / (rh @ v)
        s = r - alpha * v
        sh = M(s)
        t = A @ sh
        omega = (t @ s) / (t @ t)
        x = x + alpha * ph + omega * sh
        r = s - omega * t
        rho = rho1
    return x


@pytest.mark.parametrize("steps", [1, 2, 3, 5])
def test_bicgstab_iterates(steps):
    A, cfg, h, b = system()
    O = oracle.OracleHierarchy(h)
    ref = bicgstab(A, lambda r: O.cycle(np.zeros_like(r), r), b, steps)
    for _ in range(3):  # launched directly, captured, replayed
        x, it, rel = draugr.bicgstab(np.zeros_like(b), b, h, cfg, tol=1e-14, maxiter=steps)
        assert it == steps
        # rounding grows with the steps' condition; 1e-12 per step measured
        assert np.linalg.norm(x - ref) < 1e-10 * np.linalg.norm(ref)
        assert abs(rel - np.linalg.norm(b - A @ x) / np.linalg.norm(b)) < 1e-12


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("transpose", [False, True])
def test_bicgstab_from_the_solution(transpose, precision):
    """No residual at the start and a tolerance of zero: the solve ends on the
    breakdown test and leaves x as it was."""
    A = problems.poisson2d(12)
    cfg = draugr.hypre_default_config(smoother=draugr.L1JacobiSmootherType())
    h = draugr.amg_setup(A, cfg)
    xs = np.random.default_rng(0).integers(-4, 5, A.shape[0]).astype(float)  # whole numbers: b is exact
    x, it, rel = draugr.bicgstab(xs.copy(), A @ xs, h, cfg, tol=0.0, maxiter=5, transpose=transpose,
                                 precision=precision)
    assert np.array_equal(x, xs) and rel == 0.0 and it == 1


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("restart,maxiter", [(1, 3), (3, 3), (3, 7), (30, 4)])
def test_fgmres_stops_where_asked(restart, maxiter, precision):
    A, cfg, h, b = system()
    xs = []
    for _ in range(2):
        x, it, rel = draugr.fgmres(np.zeros_like(b), b, h, cfg, tol=1e-14, maxiter=maxiter, restart=restart,
                                   precision=precision)
        assert it == maxiter
        assert abs(rel - np.linalg.norm(b - A @ x) / np.linalg.norm(b)) < 1e-12
        xs.append(x)
    assert np.array_equal(xs[0], xs[1])
    x, it, rel = draugr.fgmres(np.zeros_like(b), b, h, cfg, tol=1e-9, maxiter=200, restart=restart,
                               precision=precision)
    assert rel < 1e-9 and it < 200


@pytest.mark.parametrize("coarse", [3, 32, 33, 64, 90])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_transposed_solve(coarse, precision):
    A, cfg, h, b = system(coarse=coarse)
    x, it, rel = draugr.bicgstab(np.zeros_like(b), b, h, cfg, tol=1e-10, maxiter=200, transpose=True,
                                 precision=precision)
    assert it < 60
    assert np.linalg.norm(b - A.T @ x) < 1e-9 * np.linalg.norm(b)

"""BiCGStab and FGMRES with their scalars on the device: iterates after a few
steps against NumPy with the oracle's cycle as the preconditioner, solves that
stop by their tolerance with the next step already enqueued (which must not
change x), and the transposed coarsest solve at the edges of its kernels."""

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
    """Per step: the iterate after its half step and after it, and the
    relative norms of s and r."""
    x, r = np.zeros_like(b), b.copy()
    rh, p, v = r.copy(), np.zeros_like(b), np.zeros_like(b)
    rho = alpha = omega = 1.0
    out, bn = [], np.linalg.norm(b)
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
        half = x + alpha * ph
        x = half + omega * sh
        r = s - omega * t
        rho = rho1
        out.append((half, x, np.linalg.norm(s) / bn, np.linalg.norm(r) / bn))
    return out


@pytest.mark.parametrize("steps", [1, 2, 3, 5])
def test_bicgstab_iterates(steps):
    A, cfg, h, b = system()
    O = oracle.OracleHierarchy(h)
    ref = bicgstab(A, lambda r: O.cycle(np.zeros_like(r), r), b, steps)[-1][1]
    for _ in range(3):  # launched directly, captured, replayed
        x, it, rel = draugr.bicgstab(np.zeros_like(b), b, h, cfg, tol=1e-14, maxiter=steps)
        assert it == steps
        # rounding grows with the steps' condition; 1e-12 per step measured
        assert np.linalg.norm(x - ref) < 1e-10 * np.linalg.norm(ref)
        assert abs(rel - np.linalg.norm(b - A @ x) / np.linalg.norm(b)) < 1e-12


@pytest.mark.parametrize("half", [False, True], ids=["full_step", "half_step"])
def test_bicgstab_stops_with_a_step_enqueued(half):
    """A tolerance that step k meets first, at its end or at its half: the
    step enqueued behind it leaves x alone."""
    A, cfg, h, b = system()
    O = oracle.OracleHierarchy(h)
    steps = bicgstab(A, lambda r: O.cycle(np.zeros_like(r), r), b, 9)
    norms = [v for st in steps for v in st[2:]]  # in the order the tests see them
    pick = [i for i in range(2 if half else 3, len(norms), 2) if norms[i] < 0.6 * min(norms[:i])]
    assert pick
    for i in pick:
        k, tol = i // 2 + 1, 1.2 * norms[i]
        want = steps[k - 1][0 if half else 1]
        for _ in range(3):  # launched directly, captured, replayed
            x, it, rel = draugr.bicgstab(np.zeros_like(b), b, h, cfg, tol=tol, maxiter=50)
            assert it == k
            # rounding grows with the steps' condition; 1e-12 per step measured
            assert np.linalg.norm(x - want) < 1e-10 * np.linalg.norm(want)
            assert abs(rel - norms[i]) < 1e-8 * norms[i] + 1e-12
        if not half:  # the same solve with no step behind it
            y, it, _ = draugr.bicgstab(np.zeros_like(b), b, h, cfg, tol=tol, maxiter=k)
            assert it == k and np.array_equal(x, y)


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

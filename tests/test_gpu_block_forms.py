"""Block solves through the forms of their products: one to eight lanes per
group (k = 4 .. 32), rows split over a warp on the long-row levels, the fused
first Jacobi step and residual (one pre-smoothing step) and the separate
kernels (none, two), V and W cycles, both precisions, each column against a
single-vector solve."""

import numpy as np
import pytest
import torch

import draugr
from draugr import problems

pytestmark = pytest.mark.gpu


FORMS = [(4, 1, 1, "V"), (8, 1, 1, "W"), (12, 1, 2, "V"), (16, 2, 1, "V"), (20, 0, 2, "V"), (32, 1, 1, "V"),
         (32, 2, 2, "W"), (6, 1, 1, "V")]


def hierarchy(pre, post, cycle):
    A = problems.heterogeneous_diffusion_3d(22, seed=4)
    cfg = draugr.hypre_default_config(agg_trunc_factor=0.2, smoother=draugr.L1JacobiSmootherType(), cycle_type=cycle,
                                      pre_smoothing_steps=pre, post_smoothing_steps=post, seed=1)
    return A, A.shape[0], cfg, draugr.amg_setup(A, cfg)


def right_hand_sides(n, k):
    B = torch.rand((n, k), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3)) - 0.5
    B[:, k // 2] = 0.0  # a column that has nothing to do
    torch.cuda.synchronize()
    return B


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k,pre,post,cycle", FORMS)
def test_block_columns(k, pre, post, cycle, precision):
    A, n, cfg, h = hierarchy(pre, post, cycle)
    B = right_hand_sides(n, k)
    X = torch.zeros_like(B)
    draugr.pcg_multi(X, B, h, cfg, tol=1e-10, precision=precision)
    R = B.cpu().numpy() - A @ X.cpu().numpy()
    for c in range(k):
        bn = float(B[:, c].norm())
        if bn == 0.0:
            assert float(X[:, c].abs().max()) == 0.0
            continue
        if pre != post:
            continue  # no symmetric preconditioner: compared after a few iterations below
        assert np.linalg.norm(R[:, c]) < 1.1e-10 * bn
        if c % 7 == 0:
            x, it, _ = draugr.pcg(torch.zeros(n, dtype=torch.float64, device="cuda"), B[:, c].contiguous(), h, cfg,
                                  tol=1e-10, precision=precision)
            assert float((X[:, c] - x).norm()) < 1e-7 * float(x.norm())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k,pre,post,cycle", FORMS)
def test_block_iterates(k, pre, post, cycle, precision):
    """Two iterations, where rounding has not grown yet, against the
    single-vector solve, for every form (also those that converge slowly or
    not at all)."""
    A, n, cfg, h = hierarchy(pre, post, cycle)
    B = right_hand_sides(n, k)
    X = torch.zeros_like(B)
    draugr.pcg_multi(X, B, h, cfg, tol=0.0, maxiter=2, precision=precision)
    longest = max(int(np.diff(h.export(l, "A_rowptr")).max()) for l in range(h.nlevels))
    # sums of up to `longest` products in another order, on each level's way down and up, both iterations
    tol = (2.2e-16 if precision == "fp64" else 6e-8) * longest * 2 * h.nlevels * 2
    for c in range(0, k, 3):
        if c == k // 2:
            continue
        x, _, _ = draugr.pcg(torch.zeros(n, dtype=torch.float64, device="cuda"), B[:, c].contiguous(), h, cfg,
                             tol=0.0, maxiter=2, precision=precision)
        assert float((X[:, c] - x).norm()) < tol * float(x.norm())


def test_hierarchy_reaches_the_split_products():
    """Levels with rows of over 64 entries, few enough rows to be split over a
    warp's groups, in a hierarchy summed in a tree (over 32 entries a row on
    average): what the comparisons above rely on."""
    _, _, _, h = hierarchy(1, 1, "V")
    lengths = [np.diff(h.export(l, "A_rowptr")) for l in range(h.nlevels)]
    assert any(r.mean() > 32 for r in lengths)
    split = [len(r) for r in lengths if r.max() > 64 and len(r) * 8 <= 32 * 32 * 148]
    assert len(split) >= 3

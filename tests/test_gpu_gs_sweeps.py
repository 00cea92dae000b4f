"""Coloured Gauss-Seidel sweeps against NumPy at the sizes where their kernels
change: rows longer than a group's registers hold, colours larger than the
cluster's row groups, the largest iterate that fits in shared memory and the
first that does not, short and long rows, one and several sweeps."""

import numpy as np
import pytest
import scipy.sparse as sp

import draugr
from draugr import problems

pytestmark = pytest.mark.gpu


def long_rows(n, nlong, length):
    rng = np.random.default_rng(5)
    A = problems.poisson1d(n).tolil()
    for i in range(nlong):
        cols = rng.choice(n, size=length, replace=False)
        A[i, cols] = -0.01
        A[cols, i] = -0.01
        A[i, i] = 4.0 + 0.02 * length
    A = sp.csr_matrix(A)
    A.sort_indices()
    return A


def banded(n, width):
    """Every row coupled to the next `width` ones: width + 1 colours."""
    offs = range(-width, width + 1)
    return sp.diags([np.full(n - abs(o), 2.0 * width if o == 0 else -1.0) for o in offs], list(offs),
                    format="csr").sorted_indices()


def nine_point(m):
    """9-point stencil on m^2 nodes: 4 colours."""
    t = sp.diags([np.ones(m - 1), np.ones(m), np.ones(m - 1)], [-1, 0, 1])
    return sp.csr_matrix(9 * sp.eye(m * m) - sp.kron(t, t)).sorted_indices()


def with_long_rows(A, nlong, length):
    """Couple nlong rows, far from one another, to `length` columns each."""
    n = A.shape[0]
    rng = np.random.default_rng(6)
    rows = np.repeat(np.arange(nlong) * (n // nlong), length)
    cols = rng.choice(n, size=nlong * length, replace=False)
    C = sp.csr_matrix((np.full(len(rows), -0.01), (rows, cols)), shape=A.shape)
    C = sp.csr_matrix(C + C.T)
    C.setdiag(0)
    return sp.csr_matrix(A + C + sp.diags(np.asarray(-C.sum(1)).ravel())).sorted_indices()


def sweeps(A, order, off, invd, x, b, steps):
    x = x.copy()
    for _ in range(steps):
        for c in range(len(off) - 1):
            rows = order[off[c]:off[c + 1]]
            x[rows] += invd[rows] * (b[rows] - A[rows] @ x)
    return x


# matrix, and whether each precision's sweeps are one cluster launch
CASES = {
    "rows_700_short": (lambda: long_rows(3000, 3, 700), True, True),       # 8 lanes per row, remainder loop
    "rows_900_long": (lambda: long_rows(400, 40, 390), True, True),        # 32 lanes per row
    "poisson1d_5": (lambda: problems.poisson1d(5), True, True),
    "poisson2d_46": (lambda: problems.poisson2d(46, 44), True, True),      # 2 colours of 1012 rows
    "poisson2d_47": (lambda: problems.poisson2d(47, 46), False, False),    # of 1081: a launch per colour
    "fe27_15": (lambda: problems.anisotropic_27pt(15), True, True),        # 8 colours of about 420 rows
    "banded_27000": (lambda: banded(27000, 115), True, True),              # 116 colours: FP64 iterate just fits
    "banded_29100": (lambda: banded(29100, 115), False, True),             # it does not
}


def launched(lib, h, x, b, steps, prec):
    before = lib.draugr_b200_kernel_launches()
    got = h.level_op(0, 2, x, b, steps=steps, precision=prec)
    return got, lib.draugr_b200_kernel_launches() - before


@pytest.mark.parametrize("smoother", [draugr.ColoredGaussSeidelType, draugr.L1ColoredGaussSeidelType])
@pytest.mark.parametrize("name", list(CASES))
def test_gs_sweeps(name, smoother):
    make, *cluster = CASES[name]
    A = make()
    n = A.shape[0]
    h = draugr.amg_setup(A, draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25), smoother=smoother(),
                                             max_coarse_size=2, max_levels=3))
    order, off, invd = h.export(0, "color_order"), h.export(0, "color_offsets"), h.export(0, "invdiag")
    rng = np.random.default_rng(1)
    x, b = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    longest = int(np.diff(A.indptr).max())
    lib = draugr.load()
    for prec, eps in ((0, 2.2e-16), (1, 1.2e-7)):
        h.level_op(0, 2, x, b, steps=1, precision=prec)  # the first FP32 call also converts the matrix
        count = {}
        for steps in (1, 2, 3):
            ref = sweeps(A, order, off, invd, x, b, steps)
            got, count[steps] = launched(lib, h, x, b, steps, prec)
            # a row's sum of `longest` products in another order, every sweep
            tol = 4 * eps * longest * steps
            assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref), (steps, prec)
        assert count[3] - count[1] == (0 if cluster[prec] else 2 * (len(off) - 1))


# one launch per colour: matrix, lanes per row of its kernel
COLOR_CASES = {
    "poisson1d_3000": (lambda: problems.poisson1d(3000), 1),            # a partial last block
    "poisson3d_20": (lambda: problems.poisson3d(20), 1),                # rows of 7 of the 8 a lane holds
    "rows_9_of_1": (lambda: with_long_rows(problems.poisson1d(300001), 3, 6), 1),   # one entry left over
    "nine_point_70": (lambda: nine_point(70), 2),
    "fe27_22": (lambda: problems.anisotropic_27pt(22), 4),
    "banded_41": (lambda: banded(12000, 20), 8),
    "rows_700": (lambda: with_long_rows(problems.poisson1d(100000), 3, 700), 16),    # few long rows: more lanes
    "banded_101": (lambda: banded(18000, 50), 16),
    "banded_141": (lambda: banded(20000, 70), 32),
    "rows_340": (lambda: with_long_rows(banded(20500, 70), 5, 200), 32),            # left over from 32 lanes
}


@pytest.mark.parametrize("name", list(COLOR_CASES))
def test_colour_launches(name):
    make, lanes = COLOR_CASES[name]
    A = make()
    n = A.shape[0]
    h = draugr.amg_setup(A, draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25),
                                             smoother=draugr.ColoredGaussSeidelType()))
    order, off, invd = h.export(0, "color_order"), h.export(0, "color_offsets"), h.export(0, "invdiag")
    longest = int(np.diff(A.indptr).max())
    # the dispatch rule: 1.1 mean rows held by the lanes, more for few long rows
    want = 1
    while want < 32 and 8 * want * n < 1.1 * A.nnz:
        want *= 2
    while want < 32 and longest > 8 * want and longest * 30000 > n * want * want:
        want *= 2
    assert want == lanes
    rng = np.random.default_rng(1)
    x, b = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    lib = draugr.load()
    for prec, eps in ((0, 2.2e-16), (1, 1.2e-7)):
        h.level_op(0, 2, x, b, steps=1, precision=prec)
        count = {}
        for steps in (1, 3):
            ref = sweeps(A, order, off, invd, x, b, steps)
            got, count[steps] = launched(lib, h, x, b, steps, prec)
            # a row's sum of `longest` products in another order, every sweep
            assert np.linalg.norm(got - ref) <= 4 * eps * longest * steps * np.linalg.norm(ref), (steps, prec)
        assert count[3] - count[1] == 2 * (len(off) - 1)
    h.free()

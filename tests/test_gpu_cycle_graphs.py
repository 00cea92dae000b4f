"""Cycles replayed as a graph give the launched cycle's values bit for bit:
on new buffers, before, between and after resetups, with more option sets than
a hierarchy keeps graphs for, and on another stream."""

import numpy as np
import pytest
import torch

import draugr
from draugr import problems

pytestmark = pytest.mark.gpu


def gauss_seidel_2d():
    """32 kernels on 4096 rows: calls after the first replay a graph."""
    return problems.poisson2d(64), draugr.AMGConfig(seed=3)


def jacobi_2d():
    """A dozen kernels: every call launches them."""
    return problems.poisson2d(100), draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25),
                                                     smoother=draugr.JacobiSmootherType())


def convection():
    """FGMRES steps on a deep hierarchy of Jacobi-type levels: 30 kernels."""
    kappa = np.exp(0.3 * np.random.default_rng(2).standard_normal((128, 128)))
    A, _ = problems.convection_diffusion_2d(kappa, 20.0, seed=3)
    return A, draugr.hypre_default_config(agg_trunc_factor=0.2, smoother=draugr.L1JacobiSmootherType(), seed=3)


def vectors(n, seed=0):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)


def cycle(h, cfg, x, b):
    """On new device buffers."""
    xd, bd = torch.tensor(x, device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    draugr.amg_cycle(xd, bd, h, cfg)
    return xd.cpu().numpy()


@pytest.mark.parametrize("make", [gauss_seidel_2d, jacobi_2d, convection])
def test_repeated_cycles(make):
    A, cfg = make()
    h = draugr.amg_setup(A, cfg)
    x, b = vectors(A.shape[0])
    first = cycle(h, cfg, x, b)
    for _ in range(3):
        assert np.array_equal(cycle(h, cfg, x, b), first)
    xh = x.copy()
    draugr.amg_cycle(xh, b, h, cfg)
    assert np.array_equal(xh, first)


@pytest.mark.parametrize("make", [gauss_seidel_2d, convection])
def test_cycles_around_resetups(make):
    A, cfg = make()
    B = A.copy()
    B.data = B.data * np.random.default_rng(1).uniform(0.9, 1.1, B.nnz)
    x, b = vectors(A.shape[0])
    fresh = draugr.amg_setup(A, cfg)
    draugr.amg_resetup(fresh, B, cfg)
    want_b = cycle(fresh, cfg, x, b)  # its first cycle: launched
    h = draugr.amg_setup(A, cfg)
    want_a = [cycle(h, cfg, x, b) for _ in range(3)][0]
    for _ in range(2):
        draugr.amg_resetup(h, B, cfg)
        assert np.array_equal(cycle(h, cfg, x, b), want_b)
        draugr.amg_resetup(h, A, cfg)
        assert np.array_equal(cycle(h, cfg, x, b), want_a)
    assert not np.array_equal(want_a, want_b)


def test_host_values_of_a_resetup_arrive():
    """The level values on the device are the ones given, on every one of many
    fresh hierarchies (the upload must be ordered before its use)."""
    A, cfg = gauss_seidel_2d()
    B = A.copy()
    B.data = B.data * np.random.default_rng(1).uniform(0.9, 1.1, B.nnz)
    x, b = vectors(A.shape[0])
    first = None
    for _ in range(30):
        h = draugr.amg_setup(A, cfg)
        before = cycle(h, cfg, x, b)
        cycle(h, cfg, x, b)
        draugr.amg_resetup(h, B, cfg)
        assert np.array_equal(h.export(0, "A_nzval"), B.data)
        got = (before, cycle(h, cfg, x, b))
        first = first or got
        assert np.array_equal(got[0], first[0]) and np.array_equal(got[1], first[1])
        h.free()


def test_more_options_than_graphs():
    A, cfg = gauss_seidel_2d()
    x, b = vectors(A.shape[0])
    cfgs = [draugr.AMGConfig(seed=3, pre_smoothing_steps=p, post_smoothing_steps=q, cycle_type=c)
            for p in (0, 1, 2) for q in (1, 2, 3) for c in ("V", "W")]
    assert len(cfgs) > 16
    h = draugr.amg_setup(A, cfg)
    first = [cycle(h, c, x, b) for c in cfgs]
    for _ in range(2):
        for c, want in zip(cfgs, first):
            assert np.array_equal(cycle(h, c, x, b), want)
    for c, want in zip(cfgs, first):  # captured and replayed one by one
        for _ in range(3):
            assert np.array_equal(cycle(h, c, x, b), want)


def test_stream_change_between_replays():
    A, cfg = gauss_seidel_2d()
    x, b = vectors(A.shape[0])
    h = draugr.amg_setup(A, cfg)
    first = cycle(h, cfg, x, b)
    for _ in range(2):
        assert np.array_equal(cycle(h, cfg, x, b), first)
    side = torch.cuda.Stream()
    for stream in (side, None, side):
        h.set_stream(stream)
        for _ in range(3):
            assert np.array_equal(cycle(h, cfg, x, b), first)
    h.set_stream(None)


@pytest.mark.parametrize("make", [jacobi_2d, convection])
def test_fgmres_repeats(make):
    """FP64 steps launched on the basis vectors (few kernels, and every
    hierarchy's first step) and replayed on the hierarchy's own agree."""
    A, cfg = make()
    b = problems.rhs(A.shape[0], 5)
    xs = []
    for _ in range(3):
        h = draugr.amg_setup(A, cfg)
        x, it, rel = draugr.fgmres(np.zeros_like(b), b, h, cfg, tol=1e-9, maxiter=100, restart=5)
        x2, it2, _ = draugr.fgmres(np.zeros_like(b), b, h, cfg, tol=1e-9, maxiter=100, restart=5)
        assert it == it2 and np.array_equal(x, x2)
        # plain aggregation needs more than 100 steps of restart 5: the residual is the returned one, to
        # the rounding of one product (5 entries a row, eps 2.2e-16)
        assert abs(rel - np.linalg.norm(b - A @ x) / np.linalg.norm(b)) < 1e-14
        xs.append(x)
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])

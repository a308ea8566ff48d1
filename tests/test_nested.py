"""The nested subspace products: the plan's two programs on the host (every index checked) against
the dense evaluation, and the FP64 kernels against the dense ones on the GPU."""
import ctypes
import os
import subprocess
import sys
import time

import numpy as np
import pytest

import sgpp_gb300 as sg

EPS = 2.0 ** -52


def _grid(dim, level, basis="linear", rounds=0, seed=0):
    make = sg.Grid.createModLinearGrid if basis == "modlinear" else sg.Grid.createLinearGrid
    grid = make(dim)
    grid.getGenerator().regular(level)
    rng = np.random.default_rng(seed)
    for _ in range(rounds):
        alpha = rng.standard_normal(grid.getSize())
        grid.getGenerator().refine(sg.SurplusRefinementFunctor(alpha, 7, 0.0))
    return grid


def _points(rng, m, dim, level):
    """Interior points, dyadic points of the finest cells, faces and corners of the cube."""
    x = rng.random((m, dim))
    x[1::5] = np.round(x[1::5] * 2 ** level) / 2 ** level
    x[2::7, 0] = 0.0
    x[3::7, dim - 1] = 1.0
    x[4::11, 0] = 2.0 ** -60
    return x


def _dense(grid, x, alpha, v):
    """(B alpha, B^T v) in FP64, every grid point for every data point, and the norms' scale."""
    st = grid.getStorage()
    lev, idx = st.level.astype(np.float64), st.index.astype(np.float64)
    mod = grid.getType() == sg.GridType.ModLinear
    b = np.ones((x.shape[0], grid.getSize()))
    for t in range(x.shape[1]):
        L, i, xt = 2.0 ** lev[:, t], idx[:, t], x[:, t][:, None]
        h = 1.0 - np.abs(L * xt - i)
        if mod:
            h = np.where(i == 1, 2.0 - L * xt, h)
            h = np.where(i == L - 1, L * xt - i + 1.0, h)
            h = np.where(L == 2, 1.0, h)
        b *= np.maximum(h, 0.0)
    return b @ alpha, b.T @ v, np.abs(b) @ np.abs(alpha), np.abs(b).T @ np.abs(v)


# regular grids from one dimension to many, level 1 (one subspace) to subspaces of 512 cells,
# grids with holes and levels of their own per dimension (refined), more subspaces than a chunk
GRIDS = [(1, 1, 0), (1, 10, 0), (2, 1, 0), (2, 9, 0), (3, 6, 0), (4, 4, 9), (5, 6, 0), (6, 3, 25),
         (9, 4, 3), (12, 3, 0), (17, 2, 2), (30, 2, 0)]


@pytest.mark.parametrize("basis", ["linear", "modlinear"])
@pytest.mark.parametrize("dim,level,rounds", GRIDS)
def test_programs_on_the_host_match_the_dense_form(lib, dim, level, rounds, basis):
    grid = _grid(dim, level, basis, rounds)
    lp, ix = grid.getStorage().getLevelIndexArraysForEval()
    rng = np.random.default_rng(dim * 10 + level)
    m, n = 48, grid.getSize()
    x = np.ascontiguousarray(_points(rng, m, dim, level + 1))
    alpha, v = rng.standard_normal(n), rng.standard_normal(m)
    out, outt = np.full(m, np.nan), np.full(n, np.nan)
    rc = lib.sgmev_nest_host(dim, n, lp.ctypes.data, ix.ctypes.data, int(basis == "modlinear"), m,
                             x.ctypes.data, alpha.ctypes.data, v.ctypes.data, out.ctypes.data,
                             outt.ctypes.data)
    assert rc == 0
    ref, reft, mag, magt = _dense(grid, x, alpha, v)
    # per product 3 roundings a dimension on either side, per sum one an addend
    tol = (6 * dim + n + m) * EPS
    assert np.all(np.abs(out - ref) <= tol * (mag + 2.0 ** dim))
    assert np.all(np.abs(outt - reft) <= tol * (magt + 2.0 ** dim))


def test_grids_without_their_ancestors(lib):
    """Level vectors whose parents are missing (a storage need not be closed), shuffled points."""
    level = np.array([[3, 1, 2], [1, 1, 1], [2, 4, 1], [3, 1, 2], [1, 3, 3]], np.int32)
    index = np.array([[5, 1, 3], [1, 1, 1], [1, 9, 1], [1, 1, 1], [1, 7, 5]], np.int32)
    grid = sg.Grid.fromArrays(level, index)
    lp, ix = grid.getStorage().getLevelIndexArraysForEval()
    rng = np.random.default_rng(5)
    x = np.ascontiguousarray(_points(rng, 60, 3, 4))
    alpha, v = rng.standard_normal(5), rng.standard_normal(60)
    out, outt = np.zeros(60), np.zeros(5)
    assert lib.sgmev_nest_host(3, 5, lp.ctypes.data, ix.ctypes.data, 0, 60, x.ctypes.data,
                               alpha.ctypes.data, v.ctypes.data, out.ctypes.data,
                               outt.ctypes.data) == 0
    ref, reft, _, _ = _dense(grid, x, alpha, v)
    np.testing.assert_allclose(out, ref, atol=100 * EPS)
    np.testing.assert_allclose(outt, reft, atol=100 * EPS)


def test_grids_the_plan_does_not_take(lib):
    """Subspaces of more than 512 cells stay on the dense kernels."""
    level, index = np.array([[11]], np.int32), np.array([[3]], np.int32)
    lp, ix = sg.Grid.fromArrays(level, index).getStorage().getLevelIndexArraysForEval()
    x, one = np.array([[0.5]]), np.ones(1)
    assert lib.sgmev_nest_host(1, 1, lp.ctypes.data, ix.ctypes.data, 0, 1, x.ctypes.data,
                               one.ctypes.data, one.ctypes.data, np.zeros(1).ctypes.data,
                               np.zeros(1).ctypes.data) == 1


def _twice():
    """A storage that holds the point (1, 1; level 2, 1) twice."""
    level = np.array([[1, 1], [2, 1], [2, 1], [2, 1], [1, 2]], np.int32)
    index = np.array([[1, 1], [1, 1], [3, 1], [1, 1], [1, 3]], np.int32)
    return sg.Grid.fromArrays(level, index)


def test_grids_with_a_point_twice_are_refused_by_the_plan(lib):
    lp, ix = _twice().getStorage().getLevelIndexArraysForEval()
    x, one = np.full((1, 2), 0.3), np.ones(5)
    assert lib.sgmev_nest_host(2, 5, lp.ctypes.data, ix.ctypes.data, 0, 1, x.ctypes.data,
                               one.ctypes.data, one.ctypes.data, np.zeros(1).ctypes.data,
                               np.zeros(5).ctypes.data) == 1


def _sparse(dim, excess):
    """Eval arrays of a grid with one point in every subspace of at most 2^excess cells."""
    rows = np.zeros((1, 0))
    for _ in range(dim):
        rows = np.concatenate([np.column_stack([rows[rows.sum(axis=1) + k <= excess],
                                                np.full((rows.sum(axis=1) + k <= excess).sum(), k)])
                               for k in range(excess + 1)])
    return np.ascontiguousarray(2.0 ** (rows + 1)), np.ones(rows.shape)


def _plan_seconds(lib, lp, ix):
    n, dim = lp.shape
    none, one, out = np.zeros((0, dim)), np.ones(n), np.zeros(n)
    t = time.process_time()
    rc = lib.sgmev_nest_host(dim, n, lp.ctypes.data, ix.ctypes.data, 0, 0, none.ctypes.data, one.ctypes.data,
                             none.ctypes.data, none.ctypes.data, out.ctypes.data)
    assert rc == 0
    return time.process_time() - t


def test_plans_take_time_in_proportion_to_the_grid(lib):
    """24,310 and 92,378 subspaces with thousands of windows, both mostly of 512 cells: building every list
    again for every count of windows took 3.9 times as long per subspace with the larger number."""
    small = min(_plan_seconds(lib, *_sparse(8, 9)) for _ in range(3))
    large = min(_plan_seconds(lib, *_sparse(10, 9)) for _ in range(3))
    assert large / 92378 < 2.5 * small / 24310


def test_plans_with_more_positions_than_indices_are_refused(lib):
    """497,420 points, one in each subspace, on 1.9e8 positions."""
    lp, ix = _sparse(13, 9)
    n = lp.shape[0]
    none, one, out = np.zeros((0, 13)), np.ones(n), np.zeros(n)
    assert (np.prod(lp, axis=1) / 2 ** 13).sum() > 2 ** 27
    assert lib.sgmev_nest_host(13, n, lp.ctypes.data, ix.ctypes.data, 0, 0, none.ctypes.data, one.ctypes.data,
                               none.ctypes.data, none.ctypes.data, out.ctypes.data) == 1


# ---- GPU -------------------------------------------------------------------------------------------
def _op(grid, x, algo, precision="double"):
    cfg = sg.OperationMultipleEvalConfiguration(
        sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA,
        parameters={"precision": precision, "algo": algo})
    return sg.createOperationMultipleEval(grid, x, cfg)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [50, 9000])
@pytest.mark.parametrize("algo", ["auto", "dense", "subspace"])
@pytest.mark.parametrize("precision,unit", [("double", EPS), ("float", 2.0 ** -24), ("df64", 2.0 ** -44)])
def test_both_copies_of_a_grid_point_count(precision, unit, algo, m):
    grid = _twice()
    rng = np.random.default_rng(1)
    x = rng.random((m, 2))
    alpha, v = np.arange(1.0, 6.0), rng.random(m) + 0.5
    op = _op(grid, x, algo, precision)
    out, outt = np.zeros(m), np.full(5, -9.0)
    op.mult(alpha, out)
    op.multTranspose(v, outt)
    ref, reft, _, _ = _dense(grid, x, alpha, v)
    # a hat of level 2 is good to 4 roundings of 1, a product to 10, and one per addend
    assert np.all(np.abs(out - ref) <= 15 * unit * np.abs(alpha).sum())
    assert np.all(np.abs(outt - reft) <= (10 + m) * unit * np.abs(v).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("basis", ["linear", "modlinear"])
@pytest.mark.parametrize("m", [1, 63, 64, 65, 1025, 40000])
@pytest.mark.parametrize("dim,level,rounds", [(1, 1, 0), (1, 10, 0), (3, 6, 0), (5, 5, 0),
                                              (6, 3, 25), (9, 4, 3), (17, 2, 2)])
def test_fp64_products_match_the_dense_kernels(dim, level, rounds, m, basis):
    grid = _grid(dim, level, basis, rounds)
    n = grid.getSize()
    rng = np.random.default_rng(m + dim)
    x = _points(rng, m, dim, level + 1)
    alpha, v = rng.standard_normal(n), rng.standard_normal(m)
    op, ref = _op(grid, x, "auto"), _op(grid, x, "dense")
    op.profile(True)
    out, outr, outt, outtr = np.zeros(m), np.zeros(m), np.zeros(n), np.zeros(n)
    op.mult(alpha, out)
    op.multTranspose(v, outt)
    assert op.profileRead(sg.SGMEV_KERNEL_MULT_NEST64)[0] == 1
    assert op.profileRead(sg.SGMEV_KERNEL_MULTT_NEST64)[0] == 1
    ref.mult(alpha, outr)
    ref.multTranspose(v, outtr)
    # 3 roundings a dimension in each product on either side, one an addend in each sum; the
    # magnitudes are those of sums of |alpha| (or |v|) over hats, at most 2^dim for ModLinear ramps
    big = 1.0 if basis == "linear" else 2.0 ** min(dim, level)
    assert np.abs(out - outr).max() <= (6 * dim + n) * EPS * big * np.abs(alpha).sum()
    assert np.abs(outt - outtr).max() <= (6 * dim + m) * EPS * big * np.abs(v).sum()
    # a range gives the bits of the full product, and a second product the same bits
    lo, hi = m // 3, m - m // 4
    part = np.full(m, -7.0)
    op.mult(alpha, part, lo, hi)
    np.testing.assert_array_equal(part[lo:hi], out[lo:hi])
    assert np.all(part[:lo] == -7.0) and np.all(part[hi:] == -7.0)
    again = np.zeros(n)
    op.multTranspose(v, again)
    np.testing.assert_array_equal(again, outt)


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite_spread_as_in_the_dense_kernels(value):
    grid = _grid(4, 4)
    n, m = grid.getSize(), 500
    rng = np.random.default_rng(3)
    x = _points(rng, m, 4, 3)
    x[7, 2] = np.nan
    x[9, 1] = -0.5
    for single in (True, False):
        alpha, v = rng.standard_normal(n), rng.standard_normal(m)
        alpha[0 if single else 5] = value
        v[11 if single else 9] = value
        got, want = [], []
        for algo, into in (("auto", got), ("dense", want)):
            op = _op(grid, x, algo)
            a, b = np.zeros(m), np.zeros(n)
            op.mult(alpha, a)
            op.multTranspose(v, b)
            into += [a, b]
        for a, b in zip(got, want):
            np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
            np.testing.assert_array_equal(np.isinf(a), np.isinf(b))


def _not_finite(grid, x, algo, precision, value, at_grid, at_data):
    n, m = grid.getSize(), x.shape[0]
    rng = np.random.default_rng(4)
    alpha, v = rng.standard_normal(n), rng.standard_normal(m)
    alpha[at_grid], v[at_data] = value, value
    op = _op(grid, x, algo, precision)
    a, b = np.zeros(m), np.zeros(n)
    op.mult(alpha, a)
    op.multTranspose(v, b)
    return a, b


@pytest.mark.gpu
@pytest.mark.parametrize("basis", ["linear", "modlinear"])
@pytest.mark.parametrize("precision", ["float", "df64"])
@pytest.mark.parametrize("dim,level,rounds,m", [(1, 3, 0, 200), (2, 4, 0, 200), (4, 2, 0, 9000), (3, 3, 2, 500),
                                                (17, 2, 0, 300)])
def test_values_that_are_not_finite_on_grids_left_to_the_dense_kernels(dim, level, rounds, m, precision, basis):
    """FP32 and float-float on small grids and beyond 16 dimensions: NaN for every point outside the
    support, as the dense kernels answer there."""
    grid = _grid(dim, level, basis, rounds)
    rng = np.random.default_rng(3)
    x = rng.random((m, dim))
    x[1::5] = np.round(x[1::5] * 2 ** level) / 2 ** level
    if basis == "linear":
        x[7, 0], x[9, dim - 1] = np.nan, -0.5
    # (1e39: not finite as FP32)
    for value, at_grid, at_data in ((np.nan, 0, 3), (np.inf, grid.getSize() - 1, 9), (-np.inf, 1, m - 1),
                                    (1e39, 2, 5)):
        got = _not_finite(grid, x, "auto", precision, value, at_grid, at_data)
        want = _not_finite(grid, x, "dense", precision, value, at_grid, at_data)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
            np.testing.assert_array_equal(np.isinf(a), np.isinf(b))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["float", "df64"])
def test_values_that_are_not_finite_on_grids_of_the_subspace_kernels(precision):
    """There a coefficient only meets the points of its support, and a value the functions of its cells."""
    grid = _grid(5, 5)
    n, m = grid.getSize(), 3000
    x = np.random.default_rng(2).random((m, 5))
    at_grid = int(np.argmax(grid.getStorage().level[:, 1]))
    a, b = _not_finite(grid, x, "auto", precision, np.nan, at_grid, 11)
    one, unit = np.zeros(n), np.zeros(m)
    one[at_grid] = unit[11] = 1.0
    ref, reft, _, _ = _dense(grid, x, one, unit)
    np.testing.assert_array_equal(np.isnan(a), ref != 0.0)
    np.testing.assert_array_equal(np.isnan(b), reft != 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("basis", ["linear", "modlinear"])
@pytest.mark.parametrize("precision,unit", [("float", 2.0 ** -24), ("df64", 2.0 ** -44)])
@pytest.mark.parametrize("m", [1, 33, 2000, 70001])
@pytest.mark.parametrize("dim,level,rounds", [(1, 1, 0), (1, 10, 0), (2, 9, 0), (3, 6, 0), (4, 3, 25),
                                              (7, 5, 0), (9, 6, 0), (12, 3, 0), (16, 3, 0), (17, 2, 2)])
def test_fp32_and_df64_mult_match_fp64(dim, level, rounds, m, precision, unit, basis):
    """One window and several (9 dimensions, level 6: more coefficients than shared memory), points
    split over warps and subspaces over CTAs (small m), runs and trees of every first dimension."""
    grid = _grid(dim, level, basis, rounds)
    n = grid.getSize()
    rng = np.random.default_rng(m + dim)
    x = _points(rng, m, dim, level + 1)
    alpha = rng.standard_normal(n)
    op, ref = _op(grid, x, "auto", precision), _op(grid, x, "auto", "double")
    op.profile(True)
    out, outr, part = np.zeros(m), np.zeros(m), np.full(m, -7.0)
    op.mult(alpha, out)
    kind = sg.SGMEV_KERNEL_MULT_NEST32 if precision == "float" else sg.SGMEV_KERNEL_MULT_NESTDF
    assert op.profileRead(kind)[0] == 1
    ref.mult(alpha, outr)
    # two roundings a factor (table entry and product), one an addend
    big = 1.0 if basis == "linear" else 2.0 ** min(dim, level)
    assert np.abs(out - outr).max() <= (4 * dim + n) * unit * big * np.abs(alpha).sum()
    op.mult(alpha, part, m // 3, m - m // 4)
    np.testing.assert_array_equal(part[m // 3:m - m // 4], out[m // 3:m - m // 4])
    v, outt, outtr, again = rng.standard_normal(m), np.zeros(n), np.zeros(n), np.zeros(n)
    op.multTranspose(v, outt)
    ref.multTranspose(v, outtr)
    assert np.abs(outt - outtr).max() <= (4 * dim + m) * unit * big * np.abs(v).sum()
    op.multTranspose(v, again)
    np.testing.assert_array_equal(again, outt)
    kind = sg.SGMEV_KERNEL_MULTT_NEST32 if precision == "float" else sg.SGMEV_KERNEL_MULTT_NESTDF
    assert m > 8192 or op.profileRead(kind)[0] == 2


@pytest.mark.gpu
@pytest.mark.parametrize("dim,level,m", [(2, 3, 1), (2, 3, 8191), (2, 3, 8192), (2, 3, 8193),
                                         (9, 4, 10766), (9, 4, 10767), (9, 4, 10768),
                                         (6, 6, 1661), (6, 6, 1662), (6, 7, 5)])
def test_host_vectors_read_in_place_and_copied(dim, level, m):
    """Whole products of small host vectors against the same product asked for as two ranges, which
    go through copies: results of up to 8,192 entries, up to 12,286 entries in all."""
    grid = _grid(dim, level)
    n = grid.getSize()
    rng = np.random.default_rng(m)
    op = _op(grid, _points(rng, m, dim, level), "auto")
    alpha, v = rng.standard_normal(n), rng.standard_normal(m)
    out, outt, parts, partst = np.zeros(m), np.zeros(n), np.zeros(m), np.zeros(n)
    for _ in range(2):
        op.mult(alpha, out)
        op.multTranspose(v, outt)
        for a, b in ((0, (m + 1) // 2), ((m + 1) // 2, m)):
            op.mult(alpha, parts, a, b)
        for a, b in ((0, (n + 1) // 2), ((n + 1) // 2, n)):
            op.multTranspose(v, partst, a, b)
        np.testing.assert_array_equal(out, parts)
        np.testing.assert_array_equal(outt, partst)
        alpha, v = -2.0 * alpha, 3.0 * v


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [sg.SGMEV_SOLVE_MIXED, sg.SGMEV_SOLVE_MIXED_NATIVE64])
@pytest.mark.parametrize("dim,level,m,lam,inner", [
    (1, 1, 5, 1e-3, None),       # one direction spans everything
    (2, 3, 1, 1e-3, None), (3, 4, 700, 1e-4, None), (3, 4, 700, 1e-4, "1e-9"),
    (4, 6, 3000, 1e-7, None),    # more steps than directions are kept
    (2, 11, 2000, 1e-5, None),   # dot products in two pieces
    (1, 12, 3000, 1e-4, None), (7, 5, 3000, 1e-4, None),  # 4,095 and 4,159 entries: one cluster or not
    (5, 5, 40000, 1e-4, "0.3")])  # many short solves
def test_fits_on_kept_directions_reach_their_residual(dim, level, m, lam, inner, mode):
    grid = _grid(dim, level)
    n = grid.getSize()
    rng = np.random.default_rng(dim * level)
    x = rng.beta(2.0, 4.0, (m, dim))
    y = np.sin(4.0 * x.sum(axis=1)) + 0.1 * rng.standard_normal(m)
    op = sg.OperationMultiEvalCuda(grid, x, sg.SGMEV_FP64, {"inner_tol": inner} if inner else {})
    eps = 1e-8
    alpha, its, _ = op.fit(y, lam, 20000, eps, mode=mode)
    ref = _op(grid, x, "dense")
    b, pred, a = np.zeros(n), np.zeros(m), np.zeros(n)
    ref.multTranspose(y, b)
    ref.mult(alpha, pred)
    ref.multTranspose(pred, a)
    # the fit's own criterion, and a relative 1e-11 of the terms for the two evaluations of it
    r = b - a - lam * m * alpha
    assert np.linalg.norm(r) <= eps * np.linalg.norm(b) + 1e-11 * (np.linalg.norm(a) + np.linalg.norm(b))
    assert 0 < its < 20000


@pytest.mark.gpu
@pytest.mark.parametrize("inner,solves", [(None, 2), ("1e-7", 1)])
def test_inner_tolerances_below_the_default_floor_are_honoured(inner, solves):
    """To 1e-5 by default, so that a fit to 2e-6 takes two inner solves; asked for more, one."""
    grid = _grid(3, 4)
    rng = np.random.default_rng(12)
    x = rng.random((2000, 3))
    y = np.sin(4.0 * x.sum(axis=1)) + 0.1 * rng.standard_normal(2000)
    op = sg.OperationMultiEvalCuda(grid, x, sg.SGMEV_FP64, {"inner_tol": inner} if inner else {})
    op.profile(True)
    _, _, residual = op.fit(y, 1e-2, 1000, 2e-6, mode=sg.SGMEV_SOLVE_MIXED)
    b = np.zeros(grid.getSize())
    op.multTranspose(y, b)
    assert residual <= (2e-6 * np.linalg.norm(b)) ** 2 * (1 + 1e-6)
    # a residual product after every solve (the first one starts from 0)
    assert op.profileRead(sg.SGMEV_KERNEL_MULT_NESTDF)[0] == solves


@pytest.mark.gpu
@pytest.mark.parametrize("dim,level,m,lam", [(5, 5, 3000, 1e-7), (6, 4, 3000, 1e-8)])
def test_solves_that_fill_the_kept_directions_take_fewer_steps_than_the_recurrence(dim, level, m, lam):
    """Inner solves that end for standing still with every slot taken, and others that start from what
    they kept: kept directions whose products are another's cost more steps than the two-term recurrence
    of the plain FP64 fit (d=6, level 4: 4,471 against 4,009)."""
    grid = _grid(dim, level)
    rng = np.random.default_rng(dim * level)
    x = rng.beta(2.0, 4.0, (m, dim))
    y = np.sin(4.0 * x.sum(axis=1)) + 0.1 * rng.standard_normal(m)
    op = _op(grid, x, "auto")
    _, plain, _ = op.fit(y, lam, 20000, 1e-8, mode=sg.SGMEV_SOLVE_PLAIN)
    _, mixed, _ = op.fit(y, lam, 20000, 1e-8, mode=sg.SGMEV_SOLVE_MIXED)
    assert 128 < mixed < plain


@pytest.mark.gpu
@pytest.mark.parametrize("dim,level,m,lam", [(2, 3, 40, 1e-3), (4, 5, 3000, 1e-4), (4, 5, 3000, 1e-7)])
def test_block_fits_on_kept_directions_reach_their_residuals(dim, level, m, lam):
    """Columns that end at different steps, a zero one and two equal ones; more steps than are kept."""
    grid = _grid(dim, level)
    n, K = grid.getSize(), sg.SGMEV_BLOCK_RHS
    rng = np.random.default_rng(m)
    x = rng.beta(2.0, 4.0, (m, dim))
    y = np.stack([np.sin((k + 1.0) * x.sum(axis=1)) + 0.1 * rng.standard_normal(m) for k in range(K)])
    y[3], y[5] = 0.0, y[4]
    op = sg.OperationMultiEvalCuda(grid, x, sg.SGMEV_FP64, {"algo": "subspace"})
    eps = 1e-8
    alpha, its, _ = op.fitBlock(y, lam, 20000, eps)
    ref = _op(grid, x, "dense")
    for k in range(K):
        b, pred, a = np.zeros(n), np.zeros(m), np.zeros(n)
        ref.multTranspose(y[k], b)
        ref.mult(alpha[k], pred)
        ref.multTranspose(pred, a)
        r = b - a - lam * m * alpha[k]
        # the fit's own criterion, and a relative 1e-11 of the terms for the two evaluations of it
        assert np.linalg.norm(r) <= eps * np.linalg.norm(b) + 1e-11 * (np.linalg.norm(a) + np.linalg.norm(b))
        assert (its[k] > 0) == (k != 3) and its[k] < 20000
    assert np.all(alpha[3] == 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("built", [False, True])
@pytest.mark.parametrize("precision,unit", [("double", EPS), ("float", 2.0 ** -24), ("df64", 2.0 ** -44)])
def test_products_captured_into_a_graph(precision, unit, built):
    """A first product under capture runs on kernels that build nothing, a later one as outside."""
    torch = pytest.importorskip("torch")
    grid = _grid(4, 4)
    n, m, dim = grid.getSize(), 3000, 4
    rng = np.random.default_rng(1)
    op = _op(grid, _points(rng, m, dim, 5), "auto", precision)
    a, v = torch.from_numpy(rng.standard_normal(n)).cuda(), torch.from_numpy(rng.standard_normal(m)).cuda()
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (m, n)]
    stream = torch.cuda.Stream()
    op.setStream(stream.cuda_stream)

    def products():
        op.multDevice(a.data_ptr(), out[0].data_ptr())
        op.multTransposeDevice(v.data_ptr(), out[1].data_ptr())

    if built:
        products()
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        products()
    graph.replay()
    torch.cuda.synchronize()
    got = [o.clone() for o in out]
    products()
    torch.cuda.synchronize()
    for g, o, x, k in zip(got, out, (a, v), (n, m)):
        bound = 0.0 if built else (6 * dim + k) * unit * float(x.abs().sum())
        assert float((g - o).abs().max()) <= bound


@pytest.mark.gpu
@pytest.mark.parametrize("dim,level", [(4, 4), (10, 5), (3, 9)])
def test_single_precision_transposes_of_double_and_single_vectors(dim, level):
    """A single-precision operator's own product (double vector), then its fit's inner products (single
    vectors) on the same plan, and the product again."""
    grid = _grid(dim, level)
    n, m = grid.getSize(), 2000
    rng = np.random.default_rng(5)
    op = _op(grid, _points(rng, m, dim, 5), "auto", "float")
    v, first, again = rng.standard_normal(m), np.zeros(n), np.zeros(n)
    op.multTranspose(v, first)
    _, its, _ = op.fit(v, 1e-2, 500, 1e-8, mode=sg.SGMEV_SOLVE_MIXED)
    op.multTranspose(v, again)
    assert 0 < its < 500
    np.testing.assert_array_equal(first, again)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["double", "float", "df64"])
def test_plans_follow_the_operator_to_another_stream(precision):
    """Plans and tables built by products on a stream that is destroyed before the next grid is staged."""
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    rt = torch.cuda.cudart()
    grid = _grid(4, 4)
    m = 9000
    rng = np.random.default_rng(8)
    x = rng.random((m, 4))
    op = _op(grid, x, "auto", precision)
    first, second = ctypes.c_void_p(0), ctypes.c_void_p(0)
    assert int(rt.cudaStreamCreate(ctypes.addressof(first))) == 0
    assert int(rt.cudaStreamCreate(ctypes.addressof(second))) == 0
    op.setStream(first.value)
    for _ in range(2):
        n = grid.getSize()
        alpha, v = rng.standard_normal(n), rng.standard_normal(m)
        out, outt = np.zeros(m), np.zeros(n)
        op.mult(alpha, out)
        op.multTranspose(v, outt)
        op.fit(v, 1e-3, 100, 1e-6, mode=sg.SGMEV_SOLVE_MIXED)
        ref, reft, _, _ = _dense(grid, x, alpha, v)
        unit = {"double": EPS, "float": 2.0 ** -24, "df64": 2.0 ** -44}[precision]
        assert np.abs(out - ref).max() <= 100 * unit * np.abs(alpha).sum()
        assert np.abs(outt - reft).max() <= 100 * unit * np.abs(v).sum()
        if first.value:
            op.setStream(second.value)
            op.synchronize()
            assert int(rt.cudaStreamDestroy(first.value)) == 0
            first.value = None
        grid.getGenerator().refine(sg.SurplusRefinementFunctor(alpha, 5, 0.0))
        op.prepare()
    op.close()
    assert int(rt.cudaStreamDestroy(second.value)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("precision,unit", [("float", 2.0 ** -24), ("df64", 2.0 ** -44)])
def test_subspace_without_materialised_products_evaluates_on_the_fly(precision, unit):
    grid = _grid(4, 5)
    n, m = grid.getSize(), 3000
    rng = np.random.default_rng(6)
    x = rng.random((m, 4))
    op = sg.createOperationMultipleEval(grid, x, sg.OperationMultipleEvalConfiguration(
        sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA,
        parameters={"precision": precision, "algo": "subspace", "materialize": "off"}))
    op.profile(True)
    alpha, v, out, outt = rng.standard_normal(n), rng.standard_normal(m), np.zeros(m), np.zeros(n)
    op.mult(alpha, out)
    op.multTranspose(v, outt)
    kinds = {"float": (sg.SGMEV_KERNEL_MULT_SUB32, sg.SGMEV_KERNEL_MULTT_SUB32),
             "df64": (sg.SGMEV_KERNEL_MULT_SUBDF, sg.SGMEV_KERNEL_MULTT_SUBDF)}[precision]
    assert [op.profileRead(k)[0] for k in kinds] == [1, 1]
    ref, reft, _, _ = _dense(grid, x, alpha, v)
    # a hat of level 5 is good to 2^5 roundings of 1; sums of at most m addends
    assert np.abs(out - ref).max() <= (4 * 32 + 70) * unit * np.abs(alpha).max() * 70
    assert np.abs(outt - reft).max() <= (4 * 32 + m) * unit * np.abs(v).sum()


@pytest.mark.gpu
def test_fp32_transposes_sum_at_most_1024_points_in_fp32():
    """230,230 subspaces leave one stream of points per block; all 8,192 points at the centre, where only
    the coarsest function is not 0, with a value that a long FP32 sum rounds down every time."""
    lp, _ = _sparse(20, 6)
    grid = sg.Grid.fromArrays(np.log2(lp).astype(np.int32), np.ones(lp.shape, np.int32))
    n, m = grid.getSize(), 8192
    op = _op(grid, np.full((m, 20), 0.5), "auto", "float")
    op.profile(True)
    value = 0.5 + 2.0 ** -13 - 2.0 ** -19
    out = np.zeros(n)
    op.multTranspose(np.full(m, value), out)
    assert op.profileRead(sg.SGMEV_KERNEL_MULTT_NEST32)[0] == 1
    root = int(np.argmin(lp.sum(axis=1)))
    # sums of up to 1,024 values stay below 513: each addition rounds by at most half an ulp, 2^-16 below
    # 512, against addends of 0.5; a sum over all points loses 1.2e-4
    assert abs(out[root] - m * value) <= 2.0 ** -15 * m * value
    out[root] = 0.0
    assert np.all(out == 0.0)


SHORT_OF_MEMORY = """
import sys
sys.path.insert(0, {root!r})
import numpy as np, torch
import sgpp_gb300 as sg
grid = sg.Grid.createLinearGrid(2)
grid.getGenerator().regular(8)
n, m = grid.getSize(), 1 << 24
rng = np.random.default_rng(1)
op = sg.createOperationMultipleEval(grid, rng.random((m, 2)), sg.OperationMultipleEvalConfiguration(
    sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA))
alpha, first, second = rng.standard_normal(n), np.zeros(m), np.zeros(m)
# the tables take 2.1 GB
rest = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
op.profile(True)
op.mult(alpha, first)
assert op.profileRead(sg.SGMEV_KERNEL_MULT_NEST64)[0] == 0
assert op.profileRead(sg.SGMEV_KERNEL_MULT_FP64)[0] == 1
del rest
torch.cuda.empty_cache()
op.mult(alpha, second)
assert op.profileRead(sg.SGMEV_KERNEL_MULT_NEST64)[0] == 1
assert np.abs(first - second).max() <= (6 * 2 + n) * 2.0 ** -52 * np.abs(alpha).sum()
"""


@pytest.mark.gpu
def test_tables_refused_for_want_of_memory_are_built_once_there_is_some():
    pytest.importorskip("torch")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", SHORT_OF_MEMORY.format(root=root)], capture_output=True, text=True,
                          timeout=300)
    assert done.returncode == 0, done.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("basis", ["linear", "modlinear"])
@pytest.mark.parametrize("dim,level,rounds", [(4, 4, 6), (8, 4, 3), (8, 4, 0), (12, 3, 0)])
def test_fp32_mult_is_as_close_as_the_one_of_stored_products(dim, level, rounds, basis):
    """60,001 points, so that a thread adds all subspaces of its point in FP32; stored products are rounded
    to FP32 once. Errors against FP64 vary by some 10 % between coefficient vectors: the mean of three."""
    grid = _grid(dim, level, basis, rounds)
    n, m = grid.getSize(), 60001
    rng = np.random.default_rng(m)
    x = rng.random((m, dim))
    stored = sg.createOperationMultipleEval(grid, x, sg.OperationMultipleEvalConfiguration(
        sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA,
        parameters={"precision": "float", "algo": "subspace", "materialize": "on"}))
    nested, exact = _op(grid, x, "auto", "float"), _op(grid, x, "auto")
    errors = np.zeros(2)
    for _ in range(3):
        alpha, ref = rng.standard_normal(n), np.zeros(m)
        exact.mult(alpha, ref)
        for k, op in enumerate((nested, stored)):
            out = np.zeros(m)
            op.mult(alpha, out)
            errors[k] += np.linalg.norm(out - ref) / np.linalg.norm(ref) / 3.0
    assert errors[0] <= 1.1 * errors[1]


@pytest.mark.gpu
def test_fp32_transpose_is_as_close_as_the_one_of_stored_products():
    """Many small factors of a product, each rounded to FP32 (1.22 times the stored products' error with v_j,
    H_1 and their product rounded one by one). The mean of six vectors, within 15 %."""
    grid = _grid(8, 6)
    n, m = grid.getSize(), 8000
    rng = np.random.default_rng(1)
    x = rng.random((m, 8))
    stored = sg.createOperationMultipleEval(grid, x, sg.OperationMultipleEvalConfiguration(
        sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA,
        parameters={"precision": "float", "algo": "subspace", "materialize": "on"}))
    nested, exact = _op(grid, x, "auto", "float"), _op(grid, x, "auto")
    errors = np.zeros(2)
    for _ in range(6):
        v, ref = rng.standard_normal(m), np.zeros(n)
        exact.multTranspose(v, ref)
        for k, op in enumerate((nested, stored)):
            out = np.zeros(n)
            op.multTranspose(v, out)
            errors[k] += np.linalg.norm(out - ref) / np.linalg.norm(ref) / 6.0
    assert errors[0] <= 1.15 * errors[1]


@pytest.mark.gpu
def test_df64_mult_is_as_close_as_the_one_of_stored_products():
    """ModLinear, one tree of 16 dimensions: 1.4 times the stored products' error with one chain for all of
    its children. The mean of eight coefficient vectors, within a fifth."""
    grid = _grid(16, 3, "modlinear")
    n, m = grid.getSize(), 20000
    rng = np.random.default_rng(1)
    x = rng.random((m, 16))
    stored = sg.createOperationMultipleEval(grid, x, sg.OperationMultipleEvalConfiguration(
        sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA,
        parameters={"precision": "df64", "algo": "subspace", "materialize": "on"}))
    nested, exact = _op(grid, x, "auto", "df64"), _op(grid, x, "auto")
    errors = np.zeros(2)
    for _ in range(8):
        alpha, ref = rng.standard_normal(n), np.zeros(m)
        exact.mult(alpha, ref)
        for k, op in enumerate((nested, stored)):
            out = np.zeros(m)
            op.mult(alpha, out)
            errors[k] += np.linalg.norm(out - ref) / np.linalg.norm(ref) / 8.0
    assert errors[0] <= 1.2 * errors[1]


@pytest.mark.gpu
@pytest.mark.parametrize("basis", ["linear", "modlinear"])
@pytest.mark.parametrize("precision,unit", [("float", 2.0 ** -24), ("df64", 2.0 ** -44)])
@pytest.mark.parametrize("m", [33, 2000, 70001])
@pytest.mark.parametrize("dim,level", [(3, 6), (9, 6), (12, 3), (16, 3)])
def test_every_fp32_and_df64_result_against_its_own_addends(dim, level, m, precision, unit, basis):
    """Each result within its own roundings: a result's addends are its subspaces' (mult), or its data
    points', of which at most 1,024 are added in FP32 (multTranspose); and the error of the whole vector."""
    grid = _grid(dim, level, basis)
    n = grid.getSize()
    rng = np.random.default_rng(m + dim)
    x = _points(rng, m, dim, level + 1)
    alpha, v = rng.standard_normal(n), rng.standard_normal(m)
    op, ref = _op(grid, x, "auto", precision), _op(grid, x, "auto")
    n_sub = len(np.unique(grid.getStorage().level, axis=0))
    for product, values, size, addends in ((0, alpha, m, n_sub), (1, v, n, min(m, 1024))):
        out, exact, own = np.zeros(size), np.zeros(size), np.zeros(size)
        for o, a, into in ((op, values, out), (ref, values, exact), (ref, np.abs(values), own)):
            (o.multTranspose if product else o.mult)(a, into)
        # two roundings a factor (table entry and product) on either side of the sum
        assert np.all(np.abs(out - exact) <= (4 * dim + addends) * unit * own)
        assert np.linalg.norm(out - exact) <= (1e-6 if precision == "float" else 1e-12) * np.linalg.norm(exact)


FIRST_PRODUCT = """
import sys, time
sys.path.insert(0, {root!r})
import numpy as np
import sgpp_gb300 as sg
grid = sg.Grid.createLinearGrid(8)
grid.getGenerator().regular(4)
op = sg.createOperationMultipleEval(grid, np.random.default_rng(0).random((20000, 8)), sg.OperationMultipleEvalConfiguration(
    sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA))
out, alpha = np.zeros(20000), np.ones(grid.getSize())
t = time.perf_counter()
op.mult(alpha, out)
print(time.perf_counter() - t)
"""


@pytest.mark.gpu
def test_the_first_mult_of_a_process_loads_its_own_dimension_only():
    """0.8 ms with the plan, the tables and the kernels of one dimension, 14 to 22 with those of all; the
    dense kernel before took 1.9."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    seconds = []
    for _ in range(3):
        done = subprocess.run([sys.executable, "-c", FIRST_PRODUCT.format(root=root)], capture_output=True, text=True,
                              timeout=120)
        assert done.returncode == 0, done.stderr
        seconds.append(float(done.stdout))
    assert min(seconds) < 5e-3


@pytest.mark.gpu
@pytest.mark.parametrize("fit_first", [False, True])
@pytest.mark.parametrize("dim,level", [(6, 4), (12, 3)])
def test_single_precision_products_and_fits_where_one_block_is_the_grid(dim, level, fit_first):
    """The operator's own mult and its fits' inner one are two kernels there, each with its own launch."""
    grid = _grid(dim, level)
    n, m = grid.getSize(), 20000
    rng = np.random.default_rng(9)
    x, alpha = rng.random((m, dim)), rng.standard_normal(n)
    y = np.sin(4.0 * x.sum(axis=1)) + 0.1 * rng.standard_normal(m)
    op, ref = _op(grid, x, "auto", "float"), _op(grid, x, "auto")
    fits, outs, exact = [], [], np.zeros(m)
    for k in range(4):
        if (k % 2 == 0) == fit_first:
            fits.append(op.fit(y, 1e-3, 1000, 1e-8, mode=sg.SGMEV_SOLVE_MIXED))
        else:
            outs.append(np.zeros(m))
            op.mult(alpha, outs[-1])
    ref.mult(alpha, exact)
    np.testing.assert_array_equal(outs[0], outs[1])
    assert np.linalg.norm(outs[0] - exact) <= 1e-6 * np.linalg.norm(exact)
    np.testing.assert_array_equal(fits[0][0], fits[1][0])
    assert 0 < fits[0][1] < 1000
    double = ref.fit(y, 1e-3, 1000, 1e-10, mode=sg.SGMEV_SOLVE_PLAIN)[0]
    assert np.abs(fits[0][0] - double).max() <= 1e-5 * np.abs(double).max()

"""Small and medium fronts of given shapes, bit for bit against the oracle: two
leaf fronts of k columns and k + r rows under one dense root of order r."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_parity import assert_parity, run_both

pytestmark = pytest.mark.gpu


def arrow_system(rv, k, r, seed, kind):
    rng = np.random.default_rng(seed)
    n = 2 * k + r
    a = rng.standard_normal((n, n))
    a = a + a.T
    a[:k, k:2 * k] = 0.0
    a[k:2 * k, :k] = 0.0
    d = np.arange(2 * k)
    if kind == "delay":  # tiny diagonals: 2x2 pivots and delayed columns
        a[d, d] *= 1e-6
        a[:k, :k] *= 1e-3
    elif kind == "zero":  # an all-zero column inside a front, and ties
        a = np.sign(a) * (np.abs(a) > 0.7)
        a[k // 2, :] = 0.0
        a[:, k // 2] = 0.0
        a[2 * k:, 2 * k:] += 50.0 * np.eye(r)
    return rv.problems.from_scipy(f"arrow{k}_{r}_{kind}", a)


def check(rv, orc, k, r, kind, **opts):
    s = arrow_system(rv, k, r, 100 * k + r, kind)
    solver, ref, b = run_both(rv, orc, s, order=np.arange(s.n, dtype=np.int64), **opts)
    assert_parity(rv, s, solver, ref, b, bwd=1e-8 if kind == "zero" else 1e-12)
    solver.close()
    ref.close()


# (k, r): one column, odd sizes, warp remainders; then fronts on either side of the 27, 55, 112 and 226 KB of
# shared memory at which the launch changes, the last one too large for it
@pytest.mark.parametrize("k,r", [(1, 3), (2, 1), (5, 33), (31, 32), (31, 82), (31, 90), (31, 200), (31, 430),
                                 (31, 880), (31, 940)])
@pytest.mark.parametrize("kind", ["plain", "delay", "zero"])
def test_tpp_fronts(rv, orc, k, r, kind):
    check(rv, orc, k, r, kind, nemin=1)


# small = 0: a column of zeros is a pivot like any other (1 / 0), and the columns that it turns into NaN are zero
# pivots; both in the shared-memory and the global-memory version
@pytest.mark.parametrize("k,r", [(7, 3), (31, 32), (90, 40), (200, 30)])
def test_zero_columns_without_a_limit(rv, orc, k, r):
    s = arrow_system(rv, k, r, 7 * k + r, "plain")
    row, col = s.rowidx, np.repeat(np.arange(s.n), np.diff(s.colptr))
    zero = np.isin(row, [1, k // 2, k - 1]) | np.isin(col, [1, k // 2, k - 1])
    s.values[zero] = 0.0
    solver, ref, _ = run_both(rv, orc, s, order=np.arange(s.n, dtype=np.int64), small=0.0)
    assert solver.inertia() == ref.inertia()
    assert np.array_equal(solver.front_info()[:, :5], ref.front_info()[:, :5])
    for x, y in zip(solver.pivot_record(), ref.pivot_record()):
        assert np.array_equal(x, y, equal_nan=x.dtype == np.float64)
    solver.close()
    ref.close()


# as many fronts in a wave as change the width of their CTAs (148 multiprocessors: 128 threads above 296 fronts,
# 64 above 1184)
@pytest.mark.parametrize("count", [297, 1185])
def test_many_tpp_fronts(rv, orc, count):
    k = 13
    rng = np.random.default_rng(count)
    blocks = rng.standard_normal((count, k, k)) * (rng.random((count, 1, 1)) + 0.1)
    s = rv.problems.from_scipy("many", sp.block_diag([sp.csc_matrix(b + b.T) for b in blocks]))
    solver, ref, b = run_both(rv, orc, s, order=np.arange(s.n, dtype=np.int64))
    assert_parity(rv, s, solver, ref, b, bwd=1e-12)
    solver.close()
    ref.close()


# a small-leaf front with more than 2^31 entries (the threshold is the caller's): its pivots are all zero but
# the last, so that the factorization is a scan of 46,341 columns
def test_small_leaf_front_past_32_bit_offsets(rv):
    n = 46343
    hub = np.concatenate([[0, 1], np.arange(3, n)])
    row = np.concatenate([np.arange(n), hub, np.full(n - 1, 2)])
    col = np.concatenate([np.arange(n), np.full(n - 1, 2), hub])
    val = np.zeros(row.size)
    val[n - 1] = -2.0
    s = rv.problems.from_scipy("hub", sp.csc_matrix((val, (row, col)), shape=(n, n)))
    solver = rv.SparseLDLT.analyze(s, rv.AnalyzeOptions(rv.OrderingStrategy.USER_SUPPLIED, np.arange(n)))
    solver.factor(None, rv.FactorOptions(nemin=1, small_leaf_threshold=n))
    assert solver.stats()["max_front_size"] ** 2 > 2 ** 31
    assert solver.inertia() == (0, 1, n - 1)
    col, code, dd, _ = solver.pivot_record()
    assert np.array_equal(col, np.arange(n)) and np.all(code == 1)
    assert np.all(dd[:-1] == 0.0) and dd[-1] == -2.0
    solver.close()


@pytest.mark.parametrize("k", [40, 77, 128])
@pytest.mark.parametrize("kind", ["plain", "delay", "zero"])
def test_small_leaf_fronts(rv, orc, k, kind):
    check(rv, orc, k, 60, kind)


# 32-column blocks with and without a remainder, panels and tiles of 32 rows and one more or less
@pytest.mark.parametrize("k,r", [(32, 1), (33, 31), (63, 32), (64, 33), (65, 100), (97, 64), (300, 37)])
@pytest.mark.parametrize("kind", ["plain", "delay", "zero"])
@pytest.mark.parametrize("threshold", [2048, 10 ** 6])  # the second keeps every front on its own CTA
def test_medium_fronts(rv, orc, k, r, kind, threshold):
    check(rv, orc, k, r, kind, small_leaf_threshold=0, large_front_threshold=threshold)


# more large fronts than there are contexts for them, beside small and medium ones: the first context leaves the
# handle's stream to those and comes back to it for the root
@pytest.mark.parametrize("count", [1, 8, 9])
def test_large_fronts_beside_small_ones(rv, orc, count):
    sizes = np.array([300] * count + [70] * 6 + [20] * 6)
    r = 260
    first = np.cumsum(sizes) - sizes
    n = int(sizes.sum()) + r
    rng = np.random.default_rng(count)
    a = np.zeros((n, n))
    for f, k in zip(first, sizes):
        a[f:f + k, f:f + k] = rng.standard_normal((k, k))
        a[n - r:, f:f + k] = rng.standard_normal((r, k)) * (rng.random((r, 1)) < 0.3)
    a[n - r:, n - r:] = rng.standard_normal((r, r))
    a = a + a.T
    s = rv.problems.from_scipy("beside", a)
    solver, ref, b = run_both(rv, orc, s, order=np.arange(n, dtype=np.int64), nemin=1, small_leaf_threshold=0,
                              large_front_threshold=310)
    assert_parity(rv, s, solver, ref, b, bwd=1e-12)
    solver.close()
    ref.close()


# the medium fronts that take the large fronts' path keep FP64 updates in the mixed form
def test_routed_fronts_stay_fp64(rv):
    s = arrow_system(rv, 450, 60, 3, "plain")
    order = np.arange(s.n, dtype=np.int64)
    rec = []
    for precision in ("fp64", "mixed"):
        solver = rv.SparseLDLT.analyze(s, rv.AnalyzeOptions(rv.OrderingStrategy.USER_SUPPLIED, order))
        solver.factor(None, rv.FactorOptions(precision=precision))
        rec.append(solver.pivot_record())
        solver.close()
    for a, b in zip(*rec):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("ib,nb", [(8, 32), (17, 64), (32, 96)])
def test_medium_fronts_block_sizes(rv, orc, ib, nb):
    check(rv, orc, 150, 45, "delay", small_leaf_threshold=0, inner_block_size=ib, outer_block_size=nb)


# outer blocks whose row permutation does not fit 16 columns in a CTA's default shared memory, on fronts that the
# wave moves to the large fronts' path and on large ones
@pytest.mark.parametrize("nb", [448, 1024])
@pytest.mark.parametrize("opts", [{}, {"large_front_threshold": 600}])
def test_wide_outer_blocks(rv, orc, nb, opts):
    check(rv, orc, nb + 170, 45, "delay", outer_block_size=nb, **opts)


# every width a pass of the solve can have (8, 4, 2, 1 columns, the last one padded), over fronts of one and
# several 64-column blocks with remainders
@pytest.mark.parametrize("nrhs", [2, 3, 5, 7, 8, 9, 13])
@pytest.mark.parametrize("k,r", [(40, 23), (130, 65), (449, 64)])
def test_solve_widths(rv, orc, k, r, nrhs):
    s = arrow_system(rv, k, r, k + nrhs, "plain")
    solver, ref, b = run_both(rv, orc, s, order=np.arange(s.n, dtype=np.int64), nrhs=nrhs)
    assert_parity(rv, s, solver, ref, b, bwd=1e-12)
    solver.close()
    ref.close()


def test_solve_nan_right_hand_side(rv):
    # a NaN travels through the blocks' published values instead of looking unpublished; other columns keep theirs
    s = arrow_system(rv, 200, 70, 5, "plain")
    solver = rv.SparseLDLT.analyze(s)
    solver.factor()
    b = rv.problems.rhs_uniform(s.n, 1, 3)
    x = solver.solve(b)
    bad = b.copy(order="F")
    bad[7, 1] = np.frombuffer(b"\xff" * 8)[0]
    y = solver.solve(bad)
    assert np.isnan(y[:, 1]).any()
    for j in (0, 2):
        assert np.linalg.norm(y[:, j] - x[:, j]) <= 1e-10 * np.linalg.norm(x[:, j])
    solver.close()

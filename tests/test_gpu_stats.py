"""Per-supernode statistics (SparseLDLT::per_supernode_stats) agree with the
aggregate FactorizationStats and with the oracle's fronts."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def test_per_supernode_stats_sum_to_the_totals(rv, orc):
    s = rv.problems.kkt(8, seed=2)
    solver = rv.SparseLDLT.analyze(s)
    assert solver.per_supernode_stats() is None
    solver.factor()
    ps = solver.per_supernode_stats()
    st = solver.stats()
    assert len(ps) == st["supernodes_after_amalgamation"]
    assert sum(p["num_1x1"] for p in ps) == st["total_1x1_pivots"]
    assert sum(p["num_2x2"] for p in ps) == st["total_2x2_pivots"]
    assert sum(p["num_delayed"] for p in ps) == st["total_delayed"]
    assert max(p["front_size"] for p in ps) == st["max_front_size"]
    assert all(p["num_eliminated"] + p["num_delayed"] == p["num_fully_summed"] for p in ps)
    ref = orc.OracleFactor(s, solver.symbolic)
    assert np.array_equal(solver.front_info()[:, :5], ref.front_info()[:, :5])
    ref.close()
    solver.close()


def dense_fronts(rv, orders):
    # one front of each order: an arrow whose hub goes first fills completely
    orders = np.asarray(orders)
    first = np.cumsum(orders) - orders
    n = int(orders.sum())
    rng = np.random.default_rng(1)
    hub, leaf = np.repeat(first, orders - 1), np.delete(np.arange(n), first)
    off = rng.standard_normal(leaf.size)
    row, col = np.concatenate([np.arange(n), leaf, hub]), np.concatenate([np.arange(n), hub, leaf])
    val = np.concatenate([rng.uniform(50.0, 100.0, n), off, off])
    return rv.problems.from_scipy("fronts", sp.csc_matrix((val, (row, col)), shape=(n, n)))


# the Schur GEMMs of a wave's only large front (order 1100) are counted whatever runs beside it: small and medium
# fronts, medium fronts (order 600) that take its path, or both
@pytest.mark.parametrize("others", [[40] * 5, [600] * 3, [600] * 3 + [40] * 5])
def test_schur_gemm_counters_of_a_lone_large_front(rv, others):
    def counters(orders, profiling):
        s = dense_fronts(rv, orders)
        solver = rv.SparseLDLT.analyze(s, rv.AnalyzeOptions(rv.OrderingStrategy.USER_SUPPLIED, np.arange(s.n)))
        solver.factor()
        solver.set_profiling(profiling)
        solver.factor()
        p = solver.profile()
        assert solver.inertia()[2] == 0 and (p["syrk_ms"] > 0) == profiling
        solver.close()
        return p["syrk_launches"], p["syrk_flops"]

    alone = counters([1100], False)
    assert alone[0] > 0 and alone[1] > 0
    for profiling in (False, True):
        assert counters([1100] + others, profiling) == alone

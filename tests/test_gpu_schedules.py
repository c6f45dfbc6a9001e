"""The schedules (hpr_set_schedule) against one another: which kernels a
problem gets, and that iterates, residuals and lambda are the same to the
bit on all of them."""
import numpy as np
import pytest
import scipy.sparse as sp

from hprsocp_b200 import HPRSOCP_parameters, instances

pytestmark = pytest.mark.gpu


def _split_cones(seed, n, m, diag_q=False):
    """n variables, nearly all in cones of 65 rows (two slices and two apply
    tiles each), 3 nonzeros per row: more than 512 reduction slots on the
    variables' side for n from about 8,000."""
    rng = np.random.default_rng(seed)
    kv, kc = int(0.9 * n) // 65, m // 15
    A1 = instances._random_rows(rng, m - 5 * kc, n, np.full(m - 5 * kc, 3))
    A2 = instances._random_rows(rng, 5 * kc, n, np.full(5 * kc, 3))
    model = instances._assemble(rng, A1, A2, n - 65 * kv, [65] * kv, [5] * kc)
    if diag_q:
        model.Q = sp.diags(rng.uniform(0.0, 1.0, size=n)).tocsr()
        model.__post_init__()
    return model


@pytest.mark.parametrize("iters", [20, 50, 140])
def test_residuals_of_a_batch_past_512_slots(iters):
    """Above 512 reduction slots the residual passes add in two levels; the
    lanes that come with a cluster-resident batch add in the same order, so a
    solve reports the same residuals on both schedules, to the bit."""
    from hprsocp_b200 import Context
    model = _split_cones(1, 10000, 3000)
    res = {}
    for mode in ("auto", "engine"):
        with Context(model) as g:
            g.set_schedule(mode)
            r = g.solve(HPRSOCP_parameters(verbose=False, stoptol=1e-14, max_iter=iters))
            assert r.iter == iters
            assert r.last == g.residuals(), mode
            res[mode] = r
            g.iterate(4, True)
            assert g.last_iterate()[1] == (1 if mode == "auto" else 8)
    assert res["auto"].last == res["engine"].last
    assert np.array_equal(res["auto"].x, res["engine"].x)


@pytest.mark.parametrize("iters", [20, 50, 140])
def test_allocation_free_residuals_past_512_slots(iters):
    """hpr_compute_residuals_noalloc adds its slots as hpr_compute_residuals
    does, also where that takes two levels."""
    from hprsocp_b200 import Context
    with Context(_split_cones(1, 10000, 3000)) as g:
        g.solve(HPRSOCP_parameters(verbose=False, stoptol=1e-14, max_iter=iters))
        for bounds in (False, True):
            assert g.residuals_noalloc(bounds) == g.residuals(bounds)


@pytest.mark.parametrize("n,launches", [(60, {"auto": 1, "fused": 1, "engine": 24}),
                                        (2000, {"auto": 1, "fused": 24, "engine": 24})])
def test_each_schedule_runs_its_kernels(n, launches):
    """A problem of a few tiles runs on one CTA when that is asked for; one of
    more than 32 tiles per side then runs on the engine.  The cluster's
    shared memory is the automatic schedule's.  lambda_max(AA') comes from a
    different kernel on each and has the same bits."""
    from hprsocp_b200 import Context
    model = instances.small_socp(5 + n, n=n, diag_q=False)
    lam = {}
    for mode, count in launches.items():
        with Context(model) as g:
            g.set_schedule(mode)
            info = g.scale(HPRSOCP_parameters(verbose=False))
            lam[mode] = g.power_A()
            g.set_sigma_lambda(info["norm_b"] / info["norm_c"], 1.05 * lam[mode], 0.0)
            g.set_inner(0)
            g.iterate(12, True)
            assert g.last_iterate()[1] == count, mode
    assert lam["auto"] == lam["fused"] == lam["engine"]


@pytest.mark.parametrize("n,dim,diag_q", [(3000, 33, False), (6000, 3, False), (1500, 33, True)])
def test_a_sparse_small_problem_is_not_slower_on_the_automatic_schedule(n, dim, diag_q):
    """Two nonzeros per row: many tiles in little memory.  A cluster just large
    enough to hold them left each warp several tiles in a row and took 1.2 to
    1.6 times the engine's iteration; with one tile per warp it takes 0.6 to
    0.75 times (best of 9 batches each, in turn)."""
    from hprsocp_b200 import Context
    rng = np.random.default_rng(n + dim)
    kv, kc = n // 2 // dim, n // 6 // dim
    m2 = dim * kc
    rows = [instances._random_rows(rng, r, n, np.full(r, 2)) for r in (n // 2 - m2, m2)]
    model = instances._assemble(rng, *rows, n - dim * kv, [dim] * kv, [dim] * kc)
    if diag_q:
        model.Q = sp.diags(rng.uniform(0.0, 1.0, size=n)).tocsr()
        model.__post_init__()
    best = {"auto": np.inf, "engine": np.inf}
    with Context(model) as g:
        info = g.scale(HPRSOCP_parameters(verbose=False))
        g.set_sigma_lambda(info["norm_b"] / info["norm_c"], 1.05 * g.power_A(), 0.0)
        g.set_inner(0)
        for _ in range(9):
            for mode in best:
                g.set_schedule(mode)
                g.iterate(150, True)
                ms, launches = g.last_iterate()
                assert (launches == 1) == (mode == "auto")
                best[mode] = min(best[mode], ms)
    assert best["auto"] <= best["engine"], best


def _general_q(seed, n, per_col, row_nnz):
    """Q = B'B + D with B of `per_col` nonzeros per column in n/4 rows (about
    4 n per_col^2 nonzeros of Q), A of n/2 rows of `row_nnz` nonzeros, cones of
    20 and 25."""
    rng = np.random.default_rng(seed)
    kv, kc = n // 40, n // 150
    rows = [instances._random_rows(rng, r, n, np.full(r, row_nnz)) for r in (n // 2 - 25 * kc, 25 * kc)]
    model = instances._assemble(rng, *rows, n - 20 * kv, [20] * kv, [25] * kc)
    B = sp.csr_matrix((rng.standard_normal(per_col * n),
                       (rng.integers(0, n // 4, size=per_col * n), np.repeat(np.arange(n), per_col))),
                      shape=(n // 4, n))
    model.Q = (B.T @ B + sp.diags(rng.uniform(0.01, 1.0, size=n))).tocsr()
    model.c = model.c - model.Q @ model.planted["x0"]
    model.__post_init__()
    return model


@pytest.mark.parametrize("n,per_col,row_nnz,launches", [(2000, 5, 5, 1), (1500, 6, 10, 1), (4000, 4, 2, 48)])
def test_a_problem_of_mostly_q_that_fits_the_cluster(n, per_col, row_nnz, launches):
    """Q is kept once in the cluster's shared memory, A twice: 197,000 and
    208,000 nonzeros of Q fit 16 CTAs beside 5,000 and 7,500 of A; 259,000 and
    three copies of the vectors of n = 4000 do not."""
    from hprsocp_b200 import Context
    model = _general_q(n, n, per_col, row_nnz)
    res = {}
    for mode in ("auto", "engine"):
        with Context(model) as g:
            g.set_schedule(mode)
            info = g.scale(HPRSOCP_parameters(verbose=False))
            g.set_sigma_lambda(info["norm_b"] / info["norm_c"], 1.05 * g.power_A(), 1.05 * g.power_Q())
            g.set_inner(0)
            g.iterate(12, True)
            assert g.last_iterate()[1] == (launches if mode == "auto" else 48)
            res[mode] = [g.get(v) for v in ("x", "x_bar", "z_bar", "y", "y_bar", "s", "w", "w_bar", "ATy", "dx", "dy")]
    for a, b in zip(res["auto"], res["engine"]):
        assert np.array_equal(a, b)

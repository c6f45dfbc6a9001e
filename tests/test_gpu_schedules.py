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
    enough to hold them leaves each warp several tiles in a row and takes 1.05
    to 1.6 times the engine's iteration; with one tile per warp it takes 0.6 to
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


VECS = ["x", "x_hat", "x_bar", "z_bar", "y", "y_bar", "s", "dx", "dy"]
QVECS = VECS + ["w", "w_bar", "ATy", "dw"]


def _run(model, mode, batches=((70, True), (1, False), (30, True))):
    """Iterates after the batches, the launches of each, lambda and the
    residuals on one schedule."""
    from hprsocp_b200 import Context
    with Context(model) as g:
        g.set_schedule(mode)
        info = g.scale(HPRSOCP_parameters(verbose=False))
        lam = g.power_A()
        diag = model.Q is not None and (model.Q - sp.diags(model.Q.diagonal())).nnz == 0
        lamq = 0.0 if model.Q is None or diag else 1.05 * g.power_Q()
        g.set_sigma_lambda(info["norm_b"] / info["norm_c"], 1.05 * lam, lamq)
        g.set_inner(0)
        launches = []
        for k, full in batches:
            g.iterate(k, full)
            launches.append(g.last_iterate()[1])
        return ([g.get(v) for v in (VECS if model.Q is None else QVECS)] + [np.array(g.scalars()), np.array(lam)],
                launches, g.residuals())


def _same(a, b):
    assert a[2] == b[2]
    for u, v in zip(a[0], b[0]):
        assert np.array_equal(u, v)


# (with a diagonal Q one CTA up to n of about 400, then clusters of 2 to 16; a
# general Q on 1 to 16; cones of 65 and more are split over tiles, which adds a
# barrier in the half-steps that project)
@pytest.mark.parametrize("kind,n", [("diag", 60), ("diag", 400), ("diag", 803), ("diag", 1200), ("diag", 2000),
                                    ("general", 60), ("general", 300), ("general", 1000), ("general", 2500),
                                    ("split", 1000), ("split", 2500), ("split_diag", 1000), ("split_diag", 2500),
                                    ("split_diag", 5200)])
def test_cluster_batches_are_the_engines_to_the_bit(kind, n):
    """One launch per batch on the cluster, 2 or 4 per iteration on the engine;
    iterates, lambda and residuals the same."""
    if kind == "diag":
        model = instances.small_socp(7 + n, n=n, diag_q=True)
    elif kind == "general":
        model = instances.qp_csr(n, n=n)
    else:
        model = _split_cones(n, n, n // 2, kind == "split_diag")
    a, e = _run(model, "auto"), _run(model, "engine")
    assert a[1] == [1, 1, 1]
    per = 2 if model.Q is None else 4
    assert e[1] == [70 * per, per, 30 * per]
    _same(a, e)


@pytest.mark.parametrize("n", [1100, 1600])
@pytest.mark.parametrize("q", ["none", "general", "dense_row"])
def test_single_cta_with_a_row_longer_than_a_tile(n, q):
    """A dense budget row (and, in the last form, a dense row and column of Q)
    of more than 1024 nonzeros keeps a problem of a few tiles out of the
    cluster: it runs on one CTA, on the engine, or, at first, half on each to
    choose.  All the same to the bit, and lambda too."""
    rng = np.random.default_rng(n)
    m1, kc, kv = 40, 8, n // 40
    A1 = sp.vstack([sp.csr_matrix(rng.uniform(0.5, 1.5, size=(1, n))),
                    instances._random_rows(rng, m1 - 1, n, np.full(m1 - 1, 5))]).tocsr()
    A2 = instances._random_rows(rng, 5 * kc, n, np.full(5 * kc, 4))
    model = instances._assemble(rng, A1, A2, n - 20 * kv, [20] * kv, [5] * kc)
    if q == "general":
        B = sp.random(20, n, density=12 / n, random_state=rng, data_rvs=rng.standard_normal, format="csr")
        model.Q = (B.T @ B + sp.diags(rng.uniform(0.5, 1.0, size=n))).tocsr()
    elif q == "dense_row":
        arrow = sp.csr_matrix((np.full(n, 0.01), (np.full(n, 3), np.arange(n))), shape=(n, n))
        model.Q = (arrow + arrow.T + sp.diags(rng.uniform(1.0, 2.0, size=n))).tocsr()
    if q != "none":
        model.c = model.c - model.Q @ model.planted["x0"]
        model.__post_init__()
    f, e, a = (_run(model, mode) for mode in ("fused", "engine", "auto"))
    per = 2 if model.Q is None else 4
    assert f[1] == [1, 1, 1]
    assert e[1] == [70 * per, per, 30 * per]
    assert a[1][0] in (1, 70 * per, 1 + 35 * per)  # already chosen in this process, or half on each
    _same(f, e)
    _same(a, e)

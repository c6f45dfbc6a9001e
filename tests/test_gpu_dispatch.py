"""Iterates on both sides of the lines where the launch forms change, against
the FP64 oracle (10 iterations from zero, sigma and lambda injected; sums
regroup at most a row's parts, so 1e-12 relative)."""
import numpy as np
import pytest

from helpers import rel_err
from hprsocp_b200 import HPRSOCP_parameters, instances
from oracle_ctx import OracleContext

pytestmark = pytest.mark.gpu

VECS = ["x", "x_hat", "x_bar", "z_bar", "y", "y_bar", "s", "dx", "dy"]


def _check(model, iters=10, tol=1e-12, schedule="engine"):
    from hprsocp_b200 import Context
    with Context(model) as g:
        o = OracleContext(model, threads=0)
        p = HPRSOCP_parameters(verbose=False)
        so = o.scale(p)
        g.scale(p)
        g.set_schedule(schedule)
        lam = 1.05 * o.power_A()
        general = getattr(model, "F", None) is not None or not so["Q_is_diag"]
        lamq = 1.05 * o.power_Q() if general else 0.0
        for c in (o, g):
            c.set_sigma_lambda(so["norm_b"] / so["norm_c"], lam, lamq)
            c.set_inner(0)
            c.iterate(iters, True)
        for v in VECS:
            assert rel_err(g.get(v), o.get(v)) <= tol, v
        o.close()


@pytest.mark.parametrize("scale", [0.08, 0.1, 0.115, 0.13])
def test_one_wave_of_wide_tiles_and_more(scale):
    """About 1,600 to 2,700 tiles per side: the two-CTA form up to 2,368."""
    _check(instances.config1(3, scale=scale))


# (rows of A about n / 2, 3.5% dense: one CTA, then clusters of 2 to 16 CTAs,
# then past the largest; from about 1,100 cones are split over tiles)
@pytest.mark.parametrize("n", [50, 56, 120, 400, 690, 803, 1100, 1700, 2300, 2900, 3600])
@pytest.mark.parametrize("diag_q", [False, True])
def test_cluster_resident_batches(n, diag_q):
    _check(instances.small_socp(100 + n, n=n, diag_q=diag_q), iters=40, tol=1e-11, schedule="auto")


@pytest.mark.parametrize("n", [40, 400, 1200, 3000])
def test_cluster_resident_batches_general_q(n):
    _check(instances.qp_csr(n, n=n, density=0.02 if n < 2000 else 0.01), iters=40, tol=1e-11, schedule="auto")


@pytest.mark.parametrize("n", [60, 400, 1500])
def test_resident_and_engine_agree_to_the_bit(n):
    from hprsocp_b200 import Context
    model = instances.small_socp(7 + n, n=n, diag_q=False)
    res = []
    for mode in ("engine", "auto"):
        with Context(model) as g:
            g.set_schedule(mode)
            info = g.scale(HPRSOCP_parameters(verbose=False))
            g.set_sigma_lambda(info["norm_b"] / info["norm_c"], 1.05 * g.power_A(), 0.0)
            g.set_inner(0)
            g.iterate(70, True)
            g.iterate(1, False)
            g.iterate(30, True)
            res.append([g.get(v) for v in VECS] + [np.array(g.scalars())])
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,kind", [(50, "none"), (400, "diag"), (1100, "none"), (2600, "none"), (1200, "csr"),
                                    (3000, "csr")])
def test_residual_lanes_of_a_batch_and_resident_power(n, kind):
    """A solve's last residuals come with its last batch: they equal the
    separate residual passes over the same iterate (same sums, 1e-13 for the
    order of the slots).  lambda_max(AA') against the oracle's iteration."""
    from hprsocp_b200 import Context
    model = (instances.qp_csr(n, n=n, density=0.01) if kind == "csr"
             else instances.small_socp(31 + n, n=n, diag_q=kind == "diag"))
    p = HPRSOCP_parameters(verbose=False, stoptol=1e-14, max_iter=37)
    with Context(model) as g:
        r = g.solve(p)
        assert r.status == "MAX_ITER" and r.iter == 37
        again = g.residuals()
        for k, v in r.last.items():
            assert abs(v - again[k]) <= 1e-13 * max(1.0, abs(again[k])), (k, v, again[k])
        o = OracleContext(model, threads=0)
        o.scale(p)
        assert abs(g.power_A() - o.power_A()) <= 1e-9 * o.power_A()
        o.close()


@pytest.mark.parametrize("scale", [0.52, 0.53])
def test_gathers_through_l1_and_past_it(scale):
    """1,040,000 and 1,060,000 columns: both sides of the line (2^20) below
    which the gathers go through L1."""
    _check(instances.config1(6, scale=scale), iters=3)


@pytest.mark.parametrize("dims", [[2, 8, 3], [9, 8, 40, 3], [200, 7, 1500], [3] * 70 + [64, 65]])
def test_bound_violation_by_lane_and_by_warp(dims):
    """Cones of up to 8 rows (one lane) and above (a warp), more and fewer than
    a warp's 32: the residuals with the bound violation at a start point that
    is on both sides of every cone (norms regroup: 1e-12)."""
    from hprsocp_b200 import Context, SOCPModel
    import scipy.sparse as sp
    rng = np.random.default_rng(len(dims))
    nb, n, m = 6, 6 + sum(dims), 12
    A = sp.random(m, n, density=0.3, random_state=rng, format="csr") + sp.eye(m, n, format="csr")
    model = SOCPModel(A=A, c=rng.standard_normal(n), AL=-np.ones(m), AU=np.ones(m),
                      l=np.r_[-np.ones(nb), np.full(n - nb, -np.inf)], u=np.r_[np.ones(nb), np.full(n - nb, np.inf)],
                      soc_rhs=np.zeros(0), SOC_con_idx=np.array([m]),
                      SOC_var_idx=np.concatenate([[nb], nb + np.cumsum(dims)]), number_linear_con=m, number_lu_x=nb)
    with Context(model) as g:
        o = OracleContext(model, threads=0)
        p = HPRSOCP_parameters(verbose=False)
        o.scale(p)
        g.scale(p)
        x = 3.0 * rng.standard_normal(n)
        for c in (o, g):
            c.set("x_bar", x)
        a, b = g.residuals(True), o.residuals(True)
        for k in b:
            assert abs(a[k] - b[k]) <= 1e-12 * max(1.0, abs(b[k])), (k, a[k], b[k])
        o.close()


def test_wide_tiles_over_more_columns_than_the_l1_line():
    """600 rows of 300 nonzeros over 1,100,000 columns: the rows' side is one
    wave of wide tiles, whose gathers go through L1 at any length, the columns'
    side is past it."""
    rng = np.random.default_rng(11)
    n, kv = 1_100_000, 200
    A1 = instances._random_rows(rng, 500, n, np.full(500, 300))
    A2 = instances._random_rows(rng, 100, n, np.full(100, 300))
    _check(instances._assemble(rng, A1, A2, n - 70 * kv, [70] * kv, [5] * 20), iters=3)

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

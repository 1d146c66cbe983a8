"""Gradients through quotients and powers with the literal 1 as an operand, on
either side and in either order: the operand has no share, so nothing is kept of
the result, and the way back must not look at it.  Against the oracle's FP64
gradient, with the tolerance of test_gpu_grad.py."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")
port = pytest.importorskip("oracle.port")

OPS = ["DIV", "RDIV", "POW", "RPOW"]


@pytest.mark.parametrize("points", [1, 129, 300])
@pytest.mark.parametrize("chains", [64, 8192])
def test_operand_one(points, chains):
    """c1 + [op(u, 1) or op(1, u)] with u = c x + c', the constants positive."""
    PL = 15
    r = np.random.default_rng(points)
    x = r.uniform(0.5, 2.0, points).astype(np.float32)
    y, sd = r.uniform(1, 3, points).astype(np.float32), np.full(points, 0.5, np.float32)
    P = np.full((PL, chains), g.A, np.int32)
    C = np.ones((PL, chains), np.float32)
    P[0] = g.CPLUS
    for k in range(chains):
        op, right = getattr(g, OPS[k % 4]), (k // 4) % 2
        P[1, k] = op                                    # node 2; its children 4 and 5
        one, u = (4, 5) if right else (5, 4)
        P[one - 1, k] = g.ONE
        P[u - 1, k] = g.CPLUS
        P[2 * u - 1, k] = g.CTIMES
    C[:] = r.uniform(0.6, 1.6, C.shape).astype(np.float32)
    s = g.Sampler(chains, program_length=PL)
    try:
        s.set_data(x, y, sd)
        s.set_state(P, C)
        grad, lik = s.loglik_grad()
    finally:
        s.close()
    used = H.used_constants(P)
    for k in range(64):
        ll64, g64, gabs = port.loglik_grad_f64(P, k, C[:, k].astype(np.float64), x, y, sd)
        assert abs(lik[k] - ll64) <= 1e-5 * abs(ll64)
        assert np.all(grad[~used[:, k], k] == 0) and used[:, k].sum() == 3
        for j in np.where(used[:, k])[0]:
            assert abs(grad[j, k] - g64[j]) <= 1e-4 * abs(g64[j]) + 2e-5 * gabs[j] + 1e-18, (OPS[k % 4], j)

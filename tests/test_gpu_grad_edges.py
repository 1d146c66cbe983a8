"""The adjoint at the edges of its own layout, against the oracle's FP64
gradient with the tolerance of test_gpu_grad.py (1e-4 relative, the FP32
rounding of the sum, and four times the gradient's FP32 noise where that is
larger): programs with more constants than the shared rows take at once and
tapes longer than those in shared memory, and point counts around one pass,
an odd number of passes and a partial last one.  Then the result buffer: the
same numbers from a handle that has been called before, has run in between, or
whose results are too large to stay allocated."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")
port = pytest.importorskip("oracle.port")

REL, CANCEL, FLOOR = 1e-4, 2e-5, 1e-18


def _full_trees(P, C, seed):
    """Every even chain a full tree over the nodes: sums, products and a few
    quotients inside, a constant and the variable in turn at the leaves."""
    PL, N = P.shape
    r = np.random.default_rng(seed)
    first_leaf = (PL + 1) // 2 - 1
    for idx in range(0, N, 2):
        P[:first_leaf, idx] = r.choice([g.PLUS, g.MINUS, g.TIMES, g.DIV], first_leaf, p=[0.4, 0.2, 0.3, 0.1])
        P[first_leaf:, idx] = [g.CONST if k % 2 == 0 else g.A for k in range(PL - first_leaf)]
        C[first_leaf:, idx] = r.uniform(0.5, 1.5, PL - first_leaf).astype(np.float32)


@pytest.mark.parametrize("PL", [31, 63, 127])
@pytest.mark.parametrize("points", [1, 127, 129, 300, 640])
def test_adjoint_edges_match_fp64_gradient(PL, points):
    x, y, sd = H.rational_data(points, seed=points)
    N = 96
    P, C = H.random_programs(N, PL, ops=H.OPSET_BASIC, seed=PL + points, shallow_frac=0.0)
    _full_trees(P, C, PL * points)
    used = H.used_constants(P)
    if PL >= 63:                # a full tree has (PL + 1) / 4 constants
        assert used.sum(0).max() > 8
    s = g.Sampler(N, program_length=PL)
    try:
        s.set_data(x, y, sd)
        s.set_state(P, C)
        grad, lik = s.loglik_grad()
    finally:
        s.close()
    checked = 0
    for idx in range(N):
        c64 = C[:, idx].astype(np.float64)
        if not np.isfinite(lik[idx]) or not used[:, idx].any():
            continue
        ll64, g64, gabs = port.loglik_grad_f64(P, idx, c64, x, y, sd)
        if not np.isfinite(ll64) or abs(lik[idx] - ll64) > 1e-5 * abs(ll64):
            continue
        assert np.all(grad[~used[:, idx], idx] == 0)
        sens = None
        for k in np.where(used[:, idx])[0]:
            if not (np.isfinite(g64[k]) and np.isfinite(grad[k, idx])):
                continue
            checked += 1
            err, tol = abs(grad[k, idx] - g64[k]), REL * abs(g64[k]) + CANCEL * gabs[k] + FLOOR
            if err > tol:
                if sens is None:
                    sens = port.grad_sensitivity(P, idx, c64, x, y, sd)
                tol += 4 * sens[k]
            assert err <= tol, (idx, k, grad[k, idx], g64[k])
    assert checked > 0


@pytest.mark.parametrize("N,PL", [(1, 1), (257, 31), (270000, 127)])
def test_gradient_of_a_used_handle(N, PL):
    data = H.rational_data(65, seed=2)
    P, C = g.host_init_chains(N, PL, 9, ops=H.OPSET_BASIC)
    kw = dict(program_length=PL, ops=H.OPSET_BASIC)
    a, b = g.Sampler(N, **kw), g.Sampler(N, **kw)
    try:
        a.set_data(*data)
        a.set_state(P, C)
        first = a.loglik_grad()
        again = a.loglik_grad()
        a.run_block(3, 5)
        third = a.loglik_grad()
        b.set_data(*data)
        b.set_state(*a.get_state()[:2])
        fresh = b.loglik_grad()
    finally:
        a.close()
        b.close()
    for p, q in ((first, again), (third, fresh)):
        assert np.array_equal(p[0], q[0], equal_nan=True)
        assert np.array_equal(p[1], q[1], equal_nan=True)

"""Streamed layouts of eight points per lane, one and three input variables:
every barrier period, CTA size and kernel gives the chains of K = 4, bit for
bit; among the programs full trees, whose pending values go beyond the three
levels of the value stack that are in shared memory."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")

LAYOUTS = [(8, 0, 0, 1, 8, 0), (8, 0, 0, 1, 4, 0), (8, 0, 0, 5, 8, 0), (8, 0, 0, 0, 8, 0), (8, 0, 0, 1, 8, 1),
           (8, 0, 0, 1, 4, 1)]


def _programs(N, PL, ops, seed):
    """Random programs and, every second one, a full tree over constants and
    inputs: of sums, differences and products, or also of quotients and powers
    (many of them invalid at some point)."""
    P, C = g.host_init_chains(N, PL, seed, ops=ops)
    r = np.random.default_rng(seed)
    first_leaf = (PL + 1) // 2 - 1
    leaves = [g.CONST, g.A] + ([g.X2, g.X3] if g.X2 in ops else [])
    inner = [[g.PLUS, g.MINUS, g.PLUS, g.TIMES], [g.PLUS, g.MINUS, g.TIMES, g.DIV] + [g.POW] * (g.POW in ops)]
    for c in range(0, N, 2):
        P[:first_leaf, c] = r.choice(inner[c // 2 % 2], first_leaf)
        P[first_leaf:, c] = r.choice(leaves, PL - first_leaf)
        C[:, c] = r.uniform(0.5, 1.5, PL).astype(np.float32)
    return P, C


@pytest.mark.parametrize("nv", [1, 3])
@pytest.mark.parametrize("PL,points", [(15, 300), (127, 8193), (255, 129), (255, 2049)])
def test_eight_points_per_lane_give_the_same_chains(nv, PL, points):
    N = 77
    ops = H.OPSET_MULTI if nv == 3 else H.OPSET_BASIC
    P, C = _programs(N, PL, ops, PL + points)
    data = H.multivar_data(points, seed=points) if nv == 3 else H.expdecay_data(points, seed=points)
    res = []
    s = g.Sampler(N, program_length=PL, ops=ops, const_proposal=g.CONST_RANDOM_WALK, n_vars=nv)
    try:
        (s.set_data3 if nv == 3 else s.set_data)(*data)
        s.set_streaming(True)
        for layout in [(4, 0, 0, 1, 8, 0)] + LAYOUTS:
            s.set_layout(*layout)
            geo = s.launch_geometry()
            assert (geo["K"], geo["stream"], geo["pipe"]) == (layout[0], 1, layout[5])
            s.set_state(P, C)
            scores = s.evaluate()
            s.set_state(P, C)
            s.run_block(9, 17)
            res.append((*scores, *s.get_state()))
    finally:
        s.close()
    assert np.isfinite(res[0][1][::2]).any()
    for k, got in enumerate(res[1:]):
        for a, b in zip(res[0], got):
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), LAYOUTS[k]

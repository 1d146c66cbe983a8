"""Step-size adaptation where the acceptance ratio is not a number: the program
x has no nodes to redraw (a count of 0), so that the Hastings terms of a
structure move that keeps it, which stand until the next one, are infinite on
both sides.  Such moves are rejected, and the scale goes to its lower bound
e^-30, in every kernel."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")


@pytest.mark.parametrize("points,pipe", [(50, None), (50, 0), (50, 1), (5000, None)])
def test_scale_of_a_program_without_nodes(points, pipe):
    N, PL = 65, 7
    s = g.Sampler(N, program_length=PL, ops=[g.A, g.B], const_proposal=g.CONST_RANDOM_WALK, rw_sd=0.3)
    try:
        s.set_data(*H.quad_data(points, seed=1))
        if pipe is not None:
            s.set_layout(4, 0, 0, 1, 8, pipe)
        s.set_state(np.full((PL, N), g.A, np.int32), np.ones((PL, N), np.float32))
        s.adapt_scales(0.3)
        s.run_block(12, 5)
        scales, st = s.chain_scales(), s.stats()
    finally:
        s.close()
    assert st["const_proposed"] > 0 and st["const_accepted"] == 0
    assert np.allclose(scales, np.exp(-30.0), rtol=1e-5, atol=0)

"""The scores a block writes are those of its final programs and constants,
bit for bit, also where the kernels take a proposal's likelihood over from the
current state (a structure move of a node the program does not read, a
constant move of a program without constants): evaluating the written state
from scratch gives the same numbers."""
import numpy as np
import pytest

import gpuropolis_gb300 as g
from tests import helpers as H

pytestmark = pytest.mark.gpu

WALK, REF = g.CONST_RANDOM_WALK, g.CONST_REFERENCE


@pytest.mark.parametrize("PL", [1, 3, 31, 63, 255])
@pytest.mark.parametrize("rng,moves,ops", [(g.RNG_LCG, WALK, H.OPSET_BASIC), (g.RNG_PHILOX, REF, g.OPSET_REFERENCE),
                                           (g.RNG_LCG, WALK, [g.ONE, g.A, g.B, g.PLUS, g.DIV])])
@pytest.mark.parametrize("pipe", [0, 1])
def test_block_scores_are_those_of_the_written_state(PL, rng, moves, ops, pipe):
    N = 301
    s = g.Sampler(N, program_length=PL, ops=ops, rng=rng, const_proposal=moves, rw_sd=0.1)
    try:
        s.set_data(*H.expdecay_data(250, seed=3))
        s.set_layout(4, 0, 0, 1, 8, pipe)
        s.set_state(*g.host_init_chains(N, PL, 5, ops=ops))
        for block in range(2):
            s.run_block(37, 11 + block)
            _, _, prior, lik = s.get_state()
            prior2, lik2 = s.evaluate()
            assert np.array_equal(prior.view(np.uint64), prior2.view(np.uint64))
            assert np.array_equal(lik.view(np.uint64), lik2.view(np.uint64))
    finally:
        s.close()

"""Hamiltonian blocks with structure moves: the scores a block writes are those
of its final programs and constants, bit for bit, although a proposal that keeps
the program takes the current likelihood and gradient over and a rejected one
leaves its adjoint words behind.  Populations with many unread nodes; structure
moves at every step, every second and every fifth, one and three variables, few
chains and many (the adjoint's two widths)."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")


def _handle(N, PL, nv, eps, every, seed):
    ops = H.OPSET_MULTI if nv == 3 else H.OPSET_BASIC
    s = g.Sampler(N, program_length=PL, ops=ops, const_proposal=g.CONST_HMC, n_vars=nv)
    s.set_moves(every, eps, 3)
    (s.set_data3 if nv == 3 else s.set_data)(*(H.multivar_data if nv == 3 else H.quad_data)(300, seed=seed))
    s.set_state(*g.host_init_chains(N, PL, seed, ops=ops))
    return s


@pytest.mark.parametrize("every", [1, 2, 5])
@pytest.mark.parametrize("nv", [1, 3])
@pytest.mark.parametrize("N,PL", [(301, 31), (8192, 63), (77, 127)])
def test_block_scores_are_those_of_the_written_state(every, nv, N, PL):
    s = _handle(N, PL, nv, 0.001, every, 7)
    try:
        for block in range(2):
            s.run_block(23, 11 + block)
            _, _, prior, lik = s.get_state()
            prior2, lik2 = s.evaluate()
            assert np.array_equal(prior.view(np.uint64), prior2.view(np.uint64))
            assert np.array_equal(lik.view(np.uint64), lik2.view(np.uint64))
            assert np.isfinite(lik).mean() > 0.2
    finally:
        s.close()

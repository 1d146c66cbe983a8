"""The adjoint's two widths (one pass of 128 points per sweep with registers for
32 warps per SM, or two with registers for 16) and the rules between them: the
width that the Hamiltonian kernel reports for short and long data, few and many
chains, fixed and moving programs; and the same chains and gradients, bit for
bit, from a small population (always two passes per sweep) and from the large
one it is the beginning of, at the edges of passes, of pairs of passes and of
the gradient kernels' list of programs with long ops."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")

MANY, FEW = 8192, 96          # chains: beyond 48 per SM, within 16 (152 SMs)


def _handle(n_chains, PL, nv, points, every):
    ops = H.OPSET_MULTI if nv == 3 else H.OPSET_BASIC
    P, C = g.host_init_chains(MANY, PL, 11, ops=ops)
    s = g.Sampler(n_chains, program_length=PL, ops=ops, const_proposal=g.CONST_HMC, n_vars=nv)
    s.set_moves(every, 0.001, 3)
    (s.set_data3 if nv == 3 else s.set_data)(*(H.multivar_data if nv == 3 else H.quad_data)(points, seed=points))
    s.set_state(np.ascontiguousarray(P[:, :n_chains]), np.ascontiguousarray(C[:, :n_chains]))
    return s


@pytest.mark.parametrize("points", [1, 127, 128, 129, 257, 300, 512, 640])
@pytest.mark.parametrize("PL,nv", [(31, 1), (31, 3), (127, 1)])
def test_widths_give_the_same_chains_and_gradients(points, PL, nv):
    res = []
    for n in (FEW, MANY):
        s = _handle(n, PL, nv, points, 2)
        try:
            grad, lik = s.loglik_grad()
            s.run_block(7, 5)
            after = s.loglik_grad()
            res.append([a[..., :FEW] for a in (grad, lik, *after, *s.get_state())])
        finally:
            s.close()
    for a, b in zip(*res):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("chains,every,points,K", [
    (MANY, 5, 30, 4), (MANY, 5, 128, 4), (MANY, 5, 300, 4), (MANY, 5, 4000, 4), (MANY, 0, 128, 4), (MANY, 0, 129, 8),
    (MANY, 0, 1024, 8), (FEW, 5, 30, 8), (FEW, 5, 4000, 8), (FEW, 0, 128, 8)])
def test_hamiltonian_width(chains, every, points, K):
    """The width follows the moves, and a layout that the caller chose stays."""
    s = _handle(chains, 31, 1, points, every)
    try:
        assert s.launch_geometry()["K"] == K
        s.set_hmc_layout(2, 0)
        s.set_moves(0 if every else 5, 0.001, 3)
        s.set_moves(every, 0.001, 3)
        geo = s.launch_geometry()
        assert geo["K"] == K and geo["warps_per_cta"] == 2
    finally:
        s.close()

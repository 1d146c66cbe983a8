"""The default layout of large datasets (eight points per lane, tasks of
several passes, chunk sums beyond 64 chunks in device memory) gives the chains
of the four-points-per-lane pipelined kernel, bit for bit, at the edges of its
passes, chunks and tasks."""
import numpy as np
import pytest

import gpuropolis_gb300 as g
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,n", [(1, 4096), (1, 4097), (1, 8192), (1, 8193), (1, 8321), (1, 20001),
                                  (3, 6144), (3, 6145), (3, 8200), (3, 16385)])
@pytest.mark.parametrize("rng", [g.RNG_LCG, g.RNG_PHILOX])
def test_many_passes_give_the_same_chains(nv, n, rng):
    N, PL = 101, 63
    kw = dict(program_length=PL, ops=H.OPSET_MULTI if nv == 3 else H.OPSET_BASIC, rng=rng,
              const_proposal=g.CONST_RANDOM_WALK, n_vars=nv)
    P, C = g.host_init_chains(N, PL, 5, ops=kw["ops"])
    data = H.multivar_data(n, seed=n) if nv == 3 else H.expdecay_data(n, seed=n)
    res = []
    for default in (True, False):
        s = g.Sampler(N, **kw)
        try:
            (s.set_data3 if nv == 3 else s.set_data)(*data)
            if default:
                geo = s.launch_geometry()
                assert geo["K"] == 8 and geo["stream"] == 1 and geo["pipe"] == 0
            else:
                s.set_streaming(True)
                s.set_layout(4, 0, 0, 1, 8, 1)
            s.set_state(P, C)
            s.run_block(21, 17)
            res.append(s.get_state())
        finally:
            s.close()
    for a, b in zip(*res):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))

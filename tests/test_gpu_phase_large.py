"""gpr_debug_phase_profile on large data: the default layout (eight points per
lane, streamed, tasks of several passes) and the pipelined kernel of the same
width have phase-timed builds too, which give the layout's chains bit for bit."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")


@pytest.mark.parametrize("pipe", [0, 1])
@pytest.mark.parametrize("points", [4000, 8193, 20001])
def test_phase_profile_of_large_data(points, pipe):
    N, PL, steps = 201, 31, 11
    P, C = g.host_init_chains(N, PL, 3, ops=H.OPSET_BASIC)
    res = []
    for profile in (False, True):
        s = g.Sampler(N, program_length=PL, ops=H.OPSET_BASIC, const_proposal=g.CONST_RANDOM_WALK)
        try:
            s.set_data(*H.expdecay_data(points, seed=points))
            if pipe:
                s.set_streaming(True)
                s.set_layout(8, 0, 0, 1, 8, 1)
            geo = s.launch_geometry()
            assert (geo["K"], geo["stream"], geo["pipe"]) == (8, 1, pipe)
            s.set_state(P, C)
            if profile:
                ph = s.phase_profile(steps, 9)
                assert ph["cycles"]["evaluation"] > 0 and ph["passes"] > 0
            else:
                s.run_block(steps, 9)
            res.append(s.get_state())
        finally:
            s.close()
    for a, b in zip(*res):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))

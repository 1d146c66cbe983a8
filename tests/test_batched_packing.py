"""Many small datasets behind one handle: their arrays take at most four times
the points padded to four (CPU: the allocations of a runtime without a GPU), and
the chains of each are those of a handle that holds it alone, bit for bit, at
sizes around the lanes and chunks that a dataset's end leaves out (GPU)."""
import shutil

import numpy as np
import pytest

from tests import fake_cuda
from tests import helpers as H


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
@pytest.mark.parametrize("points", [1, 4, 12, 31, 60, 129])
def test_memory_of_small_datasets(tmp_path, points):
    fake_cuda.run(fake_cuda.link(tmp_path), """
import numpy as np
points, sets = %d, 8192
one = np.ones(points, np.float32)
s = g.Sampler(sets, program_length=3)
before = fake.fake_allocated()
s.set_batched_data([(one, one, one)] * sets)
arrays = 4 * 4 * sets * ((points + 3) // 4 * 4)          # x, y, weight, sd
assert fake.fake_allocated() - before <= 4 * arrays + 40 * sets + 4096
s.run_block(1, 1)
""" % points)


@pytest.mark.gpu
@pytest.mark.parametrize("three,hmc,stream", [(False, False, False), (False, False, True), (True, False, False),
                                              (False, True, False)])
def test_small_datasets_are_those_of_their_own_handles(three, hmc, stream):
    import gpuropolis_gb300 as g
    sizes = [1, 2, 3, 4, 5, 31, 32, 33, 127, 128, 129, 130, 159, 160, 161, 0, 1]
    cpd, PL = 8, 31
    make = H.multivar_data if three else H.quad_data
    sets = [make(n, seed=n + 1) if n else [np.zeros(0, np.float32)] * (5 if three else 3) for n in sizes]
    kw = dict(program_length=PL, ops=H.OPSET_MULTI if three else H.OPSET_BASIC, n_vars=3 if three else 1,
              const_proposal=g.CONST_HMC if hmc else g.CONST_RANDOM_WALK)
    N = cpd * len(sizes)
    P, C = g.host_init_chains(N, PL, 4, ops=kw["ops"])
    b = g.Sampler(N, **kw)
    try:
        b.set_streaming(stream)
        b.set_moves(3, 0.001, 2)
        b.set_batched_data(sets)
        b.set_state(P, C)
        b.run_block(8, 40)
        got = b.get_state()
        grad = b.loglik_grad()
    finally:
        b.close()
    for d, data in enumerate(sets):
        s = g.Sampler(cpd * (d + 1), **kw)          # the same chain numbers, of which the last are this dataset's
        try:
            s.set_moves(3, 0.001, 2)
            (s.set_data3 if three else s.set_data)(*data)
            s.set_state(np.ascontiguousarray(P[:, :s.N]), np.ascontiguousarray(C[:, :s.N]))
            s.run_block(8, 40)
            one, one_grad = s.get_state(), s.loglik_grad()
        finally:
            s.close()
        for a, w in zip((*got, *grad), (*one, *one_grad)):
            a, w = a[..., d * cpd:(d + 1) * cpd], w[..., d * cpd:]
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(w).view(np.uint8)), sizes[d]

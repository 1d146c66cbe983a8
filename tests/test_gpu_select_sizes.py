"""Device selection at the edges of its ranges: one CTA or a cluster, keys
in registers or re-read, ranks whose key is unique or shared by many chains;
against a host sort and the oracle's re-draw (bit for bit)."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")
port = pytest.importorskip("oracle.port")


@pytest.mark.parametrize("N", [31, 33, 1025, 8192, 8193, 131072, 131073, 170001])
@pytest.mark.parametrize("quantile", [0.03, 0.5, 0.999])
def test_select_and_redraw(N, quantile):
    PL = 3
    P0, C0 = g.host_init_chains(N, PL, N)
    prior, lik = H.mixed_scores(N, seed=N)
    post = prior + lik
    order = np.sort(np.where(np.isnan(post), -np.inf, post))
    s = g.Sampler(N, program_length=PL)
    try:
        s.set_state(P0, C0)
        s.set_scores(prior, lik)
        chain, best = s.map_chain()
        k = max(1, N // 100)
        top, n_top, threshold = s.top_chains(k)
        n, cut = s.resample(0, quantile, seed=N + 7)
        P1, C1, _, _ = s.get_state()
    finally:
        s.close()
    assert best == order[-1] and chain == int(np.flatnonzero(post == best)[0])
    assert threshold == order[N - k] and np.array_equal(top, np.flatnonzero(post >= threshold)) and n_top == len(top)
    n_ref, cut_ref = port.resample(port.cfg(PL=PL), P0, C0, prior, lik, 0, quantile, N + 7)
    assert n == n_ref and ((np.isnan(cut) and np.isnan(cut_ref)) or cut == cut_ref)
    assert np.array_equal(P1, P0) and np.array_equal(C1.view(np.uint32), C0.view(np.uint32))

"""What the autotuner chooses from (CPU: a runtime in which a chosen timing is
the shortest): the layout in force, which stays when nothing is faster, and for
large data, of one and of three variables, the streamed layouts of eight points
per lane with both kernels.  What it reports can be set again."""
import shutil

import pytest

from tests import fake_cuda

if shutil.which("gcc") is None:
    pytest.skip("no C compiler", allow_module_level=True)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.link(tmp_path_factory.mktemp("fake"))


SETUP = """
import numpy as np
nv, points, mode = %d, %d, %r
r = np.random.default_rng(points)
cols = [*r.normal(0, 1, (4 if nv == 3 else 2, points)).astype(np.float32), np.full(points, 0.1, np.float32)]
s = g.Sampler(16384, program_length=31, n_vars=nv, const_proposal=getattr(g, mode))
def default():
    (s.set_data3 if nv == 3 else s.set_data)(*cols)
    return s.launch_geometry()
geo = default()
fake.fake_fastest(0)
s.autotune(1, 1)
assert s.launch_geometry() == geo, (s.launch_geometry(), geo)
n = fake.fake_timings()
chosen = []
for k in range(1, n + 1):
    default()
    fake.fake_fastest(k)
    s.autotune(1, 1)
    chosen.append(s.launch_geometry())
    s.run_block(1, 1)
assert chosen[0] == geo and fake.fake_unsafe() == 0, fake.fake_why()
"""


@pytest.mark.parametrize("nv,points", [(1, 4096), (1, 8000), (1, 16384), (1, 65536), (3, 8000), (3, 65536)])
def test_large_data_are_tried_with_eight_points_per_lane(lib, nv, points):
    fake_cuda.run(lib, SETUP % (nv, points, "CONST_RANDOM_WALK") + """
assert geo["K"] == 8 and geo["stream"] == 1
got = {(c["K"], c["stream"], c["pipe"]) for c in chosen}
assert {(8, 1, 0), (8, 1, 1), (4, 1, 0), (4, 1, 1)} <= got, got
s.set_streaming(True)
for c in chosen:
    if c["stream"]:
        s.set_layout(c["K"], c["onepass"], c["rolled"], c["lockstep"], c["warps_per_cta"], c["pipe"])
        now = s.launch_geometry()
        assert all(now[v] == c[v] for v in ("K", "stream", "pipe", "lockstep", "warps_per_cta")), (now, c)
        s.run_block(1, 1)
assert fake.fake_unsafe() == 0, fake.fake_why()
""")


@pytest.mark.parametrize("nv,points", [(1, 100), (1, 250), (3, 300)])
def test_small_data_are_not(lib, nv, points):
    fake_cuda.run(lib, SETUP % (nv, points, "CONST_RANDOM_WALK") + """
assert not any(c["K"] == 8 and c["stream"] for c in chosen)
""")


@pytest.mark.parametrize("nv,points", [(1, 100), (3, 1000)])
def test_hamiltonian_layouts(lib, nv, points):
    fake_cuda.run(lib, SETUP % (nv, points, "CONST_HMC") + """
assert {c["K"] for c in chosen} == {4, 8} and {c["stream"] for c in chosen} == {0, 1}
""")


def test_refused_layouts(lib):
    fake_cuda.run(lib, """
import numpy as np
def refused(s, *layout):
    try:
        s.set_layout(*layout)
    except g.GprError as e:
        return e.code == 1
    return False
r = np.random.default_rng(0)
s = g.Sampler(128, program_length=31, n_vars=3)
s.set_data3(*r.normal(0, 1, (4, 100)).astype(np.float32), np.full(100, 0.1, np.float32))
assert refused(s, 4, 1, 0) and refused(s, 8, 1, 0) and refused(s, 8, 0, 1) and refused(s, 2, 0, 0)
s.set_layout(8, 0, 0)
assert s.launch_geometry()["stream"] == 1
b = g.Sampler(128, program_length=31)
d = [r.normal(0, 1, 50).astype(np.float32), r.normal(0, 1, 50).astype(np.float32), np.full(50, 0.1, np.float32)]
b.set_batched_data([d, d])
assert refused(b, 8, 0, 0) and refused(b, 4, 1, 0)
""")

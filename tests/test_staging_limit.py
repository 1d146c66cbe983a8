"""Data around the size at which a staged copy stops fitting beside the warps
are taken at every size (CPU: a runtime that refuses a kernel more shared memory
than its static variables leave): what does not fit is streamed."""
import shutil

import pytest

from tests import fake_cuda

if shutil.which("gcc") is None:
    pytest.skip("no C compiler", allow_module_level=True)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.link(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("PL", [31, 127, 255])
@pytest.mark.parametrize("nv", [1, 3])
def test_every_size_has_a_layout(lib, PL, nv):
    fake_cuda.run(lib, """
import numpy as np
PL, nv = %d, %d
one = np.ones(20000, np.float32)
s = g.Sampler(20000, program_length=PL, n_vars=nv)
seen = set()
for n in range(100, 18500, 60):
    d = [one[:n]] * (5 if nv == 3 else 3)
    (s.set_data3 if nv == 3 else s.set_data)(*d)
    for layout in ((4, 0, 0), (4, 0, 1), (8, 0, 0), (4, 0, 0, 1, 8, 1), (4, 0, 0, 1, 4, 0)):
        s.set_layout(*layout)
        seen.add((*layout, s.launch_geometry()["stream"]))
        s.run_block(1, 1)
assert {(4, 0, 0, 0), (4, 0, 0, 1), (4, 0, 0, 1, 8, 1, 0), (4, 0, 0, 1, 8, 1, 1)} <= seen, seen
""" % (PL, nv))

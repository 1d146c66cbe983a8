"""A call that fails part way leaves a launch layout and its kernel parameters
that belong together (CPU: a runtime whose allocations and launches fail on
demand).  Large data need rows for their chunk sums in device memory; a kernel
launched without them would write past its shared-memory board."""
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
def data(n, cols=3):
    r = np.random.default_rng(n)
    return [*r.normal(0, 1, (cols - 1, n)).astype(np.float32), np.full(n, 0.1, np.float32)]
def failing(f, mallocs=0, launches=0):
    fake.fake_fail(mallocs, launches)
    try:
        f()
    except g.GprError as e:
        return e.code
    finally:
        fake.fake_fail(0, 0)
    return 0
nv = %d
s = g.Sampler(16384, program_length=31, n_vars=nv)     # more chains than fit at once
set_data = (lambda n: s.set_data3(*data(n, 5))) if nv == 3 else (lambda n: s.set_data(*data(n)))
def block_is_safe():
    s.run_block(1, 1)
    s.sync()
    assert fake.fake_unsafe() == 0, fake.fake_why()
"""


@pytest.mark.parametrize("nv", [1, 3])
def test_new_data_without_memory_are_forgotten(lib, nv):
    """The data arrive, their rows of chunk sums do not: a block is refused, as
    on a handle without data, until data have been set."""
    fake_cuda.run(lib, SETUP % nv + """
set_data(20000)
block_is_safe()
codes = [failing(lambda: set_data(70000), mallocs=k) for k in (1, 2)]
assert codes[0] and codes[1], codes
n = fake.fake_launches()
assert failing(lambda: s.run_block(1, 1)) and fake.fake_launches() == n
set_data(70000)
block_is_safe()
""")


@pytest.mark.parametrize("nv", [1, 3])
def test_refused_layout_leaves_the_old_one(lib, nv):
    fake_cuda.run(lib, SETUP % nv + """
set_data(70000)
geo = s.launch_geometry()
for k in range(1, 4):
    if not failing(lambda: s.set_layout(4, 0, 0, 1, 8, 1), mallocs=k):
        break
    assert s.launch_geometry() == geo
    block_is_safe()
else:
    raise AssertionError("every allocation of a layout failed")
block_is_safe()
""")


@pytest.mark.parametrize("nv", [1, 3])
def test_autotuner_stopped_part_way_leaves_the_old_layout(lib, nv):
    """Each of its launches fails in turn, then each of its allocations."""
    fake_cuda.run(lib, SETUP % nv + """
set_data(70000)
geo = s.launch_geometry()
for k in range(1, 100):
    if not failing(lambda: s.autotune(1, 1), launches=k):
        break
    assert s.launch_geometry() == geo
    block_is_safe()
assert 2 < k < 99
block_is_safe()
set_data(70000)
for k in range(1, 20):
    failing(lambda: s.autotune(1, 1), mallocs=k)
    block_is_safe()
""")

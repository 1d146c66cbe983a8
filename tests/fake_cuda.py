"""The library's own objects linked against a CUDA runtime that has no GPU
(tests/fake/cudart.c), so that a test can make an allocation or a launch fail
and see what the host code does next.  Scenarios run in a process of their own."""
import ctypes
import glob
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.join(ROOT, "tests", "fake")


def link(folder):
    """The library linked against the fake runtime, in folder."""
    from gpuropolis_gb300 import build
    build.build()
    objs = [o for o in sorted(glob.glob(os.path.join(build.OBJ_DIR, "*.o")))]
    out = os.path.join(str(folder), "libfake.so")
    fake = [os.path.join(str(folder), "cudart.o"), os.path.join(str(folder), "check.o")]
    subprocess.run(["gcc", "-O1", "-fPIC", "-Wall", "-c", os.path.join(HERE, "cudart.c"), "-o", fake[0]], check=True)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INC, "-I", build.CSRC,
                    "-c", os.path.join(HERE, "check.cu"), "-o", fake[1]], check=True)
    subprocess.run(["g++", "-shared", "-o", out, *objs, *fake], check=True)
    return out


def run(lib, scenario):
    """The scenario's source, with g (the package) and fake (the runtime's
    switches) at hand, in a process of its own; what it prints."""
    src = "import sys; sys.path.insert(0, %r)\nfrom tests import fake_cuda\ng, fake = fake_cuda.load(%r)\n%s" % (
        ROOT, lib, scenario)
    r = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def load(lib):
    import gpuropolis_gb300 as g
    g.LIB_PATH = lib
    fake = ctypes.CDLL(lib)
    fake.fake_why.restype = ctypes.c_char_p
    for f in (fake.fake_launches, fake.fake_unsafe, fake.fake_clusters, fake.fake_timings):
        f.restype = ctypes.c_long
    fake.fake_allocated.restype = ctypes.c_size_t
    fake.fake_fastest.argtypes = [ctypes.c_long]
    fake.fake_fail.argtypes = [ctypes.c_long, ctypes.c_long]
    return g, fake

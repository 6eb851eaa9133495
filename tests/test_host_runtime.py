"""The host side of the library against a stand-in CUDA runtime (CPU).

tests/fake/cudart.c is preloaded in front of the runtime: device memory is host
memory, kernels do not run, and it counts what a test looks at.  Every scenario
runs in a process of its own.
"""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dbec-gp-mpi-cuda_b200")

PROLOGUE = """
import ctypes, sys
sys.path.insert(0, %r)
import gpe
fake = ctypes.CDLL(%r)
for f in ("live_bytes", "launches", "unordered", "lowered"):
    getattr(fake, "fake_" + f).restype = ctypes.c_longlong
def params(mode, n, prec=0):
    return gpe.make_params(mode, *n, .25, .25, .25, .1 * .25 ** 2, .5, 1., 1.5, .125 * min(n), precision=prec)
"""


@pytest.fixture(scope="module")
def fake(gpe_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", so, os.path.join(ROOT, "tests", "fake", "cudart.c")], check=True)

    def run(code):
        r = subprocess.run([sys.executable, "-c", PROLOGUE % (PKG, so) + code], capture_output=True, text=True,
                           timeout=300, env=dict(os.environ, LD_PRELOAD=so))
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_tables_are_in_place_before_the_next_step(fake, mode, prec):
    """Tables uploaded by gpe_create, gpe_set_tuning and gpe_autotune are ordered
    before the kernels that read them: no launch on the handle's non-blocking
    stream follows a copy on the legacy stream that nothing waited for."""
    fake("""
s = gpe.Solver(params(%d, (48, 40, 32), %d))
s.init_gaussian()
s.run(2, 50., 10.)
t = gpe.Tuning()
t.fft_max_radix = 4
s.set_tuning(t)
s.run(2, 50., 10.)
s.autotune(50., 10., nsteps=1)
s.run(2, 50., 10.)
assert fake.fake_launches() > 100
assert fake.fake_unordered() == 0, fake.fake_unordered()
""" % (mode, prec))

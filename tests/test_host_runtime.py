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
for f in ("live_bytes", "launches", "unordered", "lowered", "surplus", "device_syncs"):
    getattr(fake, "fake_" + f).restype = ctypes.c_longlong
lengths = [n for n in range(8, 1025, 2) if 2 ** 10 * 3 ** 6 * 5 ** 4 %% n == 0]  # the sides a handle takes
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


def test_a_launch_takes_no_shared_memory_from_another_handle(fake):
    """Handles of different sizes share kernels, and each may belong to a thread
    of its own: a kernel's dynamic shared memory limit is never set below what
    another handle was allowed, by steps, batch steps or operators."""
    fake("""
ok = [params(m, n, p) for n in ((8, 8, 1000), (8, 8, 64), (720, 8, 8), (40, 8, 8), (8, 1000, 8), (8, 540, 8))
      for m in (0, 1) for p in (0, 1)]
solvers = [gpe.Solver(p) for p in ok]
for s in solvers + solvers[::-1]:
    s.run(1, 50., 10.)
    s.calcluz()
for group in (ok[4:], ok[8:], ok[4:8]):
    b = gpe.Batch(group, [50.] * len(group), [10.] * len(group))
    b.run(1)
    b.close()
assert fake.fake_launches() > 100
assert fake.fake_lowered() == 0, fake.fake_lowered()
""")


def test_every_grid_a_handle_takes_steps_alone_and_in_a_batch(fake):
    """Every length a handle takes, along every axis: neither the batch's own tile
    choices (mixed-precision z lines of more than 514 points) nor a launch refuses
    it.  A launch whose dynamic bytes fit 48 KB only without the kernel's static
    ones (the batched y sweep of 144-point FP64 lines: 48512 and 944) is let
    through as any other."""
    fake("""
for n in lengths:
    for m in (0, 1):
        for shape in ((n, 8, 8), (8, n, 8), (8, 8, n)):
            for p in (0, 1) if shape[2] % 4 == 0 else (0,):
                q = params(m, shape, p)
                s = gpe.Solver(q)
                s.run(1, 50., 10., rms_every=1)
                s.close()
                b = gpe.Batch([q], [50.], [10.])
                b.run(1)
                b.close()
""")


def test_device_bytes_covers_a_handles_allocations(fake):
    """gpe_device_bytes, by which the server admits, is at least what gpe_create
    allocates, and at most 1.5 MB (its allowance for tables) and two planes of row
    sums more."""
    fake("""
for n in ((1024, 1024, 8), (1024, 512, 12), (8, 8, 1024), (8, 1024, 8), (48, 40, 32), (90, 100, 72), (8, 8, 8)):
    for m in (0, 1):
        for p in (0, 1):
            before = fake.fake_live_bytes()
            s = gpe.Solver(params(m, n, p))
            held, said = fake.fake_live_bytes() - before, gpe.device_bytes(s.params)
            assert held <= said <= held + 1.5 * 2 ** 20 + 2 * 8 * max(n[0] * n[1], n[0] * n[2], n[1] * n[2]), (n, m, p, held, said)
            s.close()
            assert fake.fake_live_bytes() == before
""")


@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_planning_again_allocates_nothing(fake, mode, prec):
    """gpe_set_tuning with no device memory left: the handle keeps its tables
    (it lost them where an allocation of the new plan failed)."""
    fake("""
s = gpe.Solver(params(%d, (48, 40, 32), %d))
held = fake.fake_live_bytes()
fake.fake_fail_mallocs(1)
for radix, seg in ((4, 8), (2, 0), (0, 0)):
    t = gpe.Tuning()
    t.fft_max_radix = radix
    t.sweep_seg[0] = seg
    s.set_tuning(t)
    s.run(1, 50., 10.)
assert fake.fake_live_bytes() == held
""" % (mode, prec))


@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_sweeps_launch_no_more_ctas_than_fit(fake, mode, prec):
    """A sweep's CTAs walk over the tiles: more of them than the SMs hold (shared
    memory, static bytes and the system's 1 KB included) would run a second
    wave behind the first."""
    fake("""
for n in (30, 60, 64, 72, 80, 96, 120, 128, 144, 180, 256, 320, 400, 500, 512, 540, 640, 750):
    for shape in ((n, 64, 64), (64, n, 64), (64, 64, n)):
        if %(p)d and shape[2] %% 4:
            continue
        q = params(%(m)d, shape, %(p)d)
        b = gpe.Batch([q] * 4, [50.] * 4, [10.] * 4)
        b.solver(0).run(1, 50., 10.)
        b.run(1)
        b.close()
        assert fake.fake_surplus() == 0, shape
""" % dict(m=mode, p=prec))


def test_no_call_waits_for_the_whole_device(fake):
    """Another thread may be capturing a batch step (the server's does): a wait for
    the device fails then and spoils the capture."""
    fake("""
for m in (0, 1):
    for p in (0, 1):
        s = gpe.Solver(params(m, (16, 12, 8), p))
        s.init_gaussian()
        s.run(2, 50., 10., rms_every=1)
        s.set_tuning(None)
        s.close()
b = gpe.Batch([params(0, (16, 12, 8))] * 2, [1., 2.], [0., 0.])
b.run(2)
b.close()
assert fake.fake_device_syncs() == 0
""")

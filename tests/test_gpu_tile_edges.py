"""The sweeps, FFT passes and observables at the sizes where their tiles and
segments can go wrong (GPU), against the oracle.

Tolerances: FP64 <= 1e-12 of the largest value, the bar of the operator tests.
Mixed precision: an operator's FP32 arithmetic is a few roundings per point
along a contracting recurrence or of log2 n stages, each 2^-24 = 6e-8; 2e-6
leaves a factor of thirty.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {0: 1e-12, 1: 2e-6}


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def pair(gpe, oracle_mod, mode, prec, n, dtf=0.1, seed=0):
    """A handle and the oracle with the same random psi (exact in FP32)."""
    dx = 0.25
    args = (*n, dx, 1.1 * dx, 0.9 * dx, dtf * dx * dx, 0.5, 1.0, 1.5, 0.5 * min(n) * dx)
    s, o = gpe.Solver(gpe.make_params(mode, *args, precision=prec)), oracle_mod.Oracle(mode, 1, *args)
    r = np.random.default_rng(seed)
    psi = r.standard_normal(n).astype(np.float32).astype(np.float64)
    if mode:
        psi = psi + 1j * r.standard_normal(n).astype(np.float32)
    s.set_psi(psi)
    o.set_psi(psi)
    return s, o, psi


# line lengths: one segment, a full last segment, every remainder class, the
# longest; time steps whose carries reach one, several and all segments
@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("n,dtf", [((8, 10, 8), .1), ((18, 36, 20), 1.), ((60, 50, 36), 3.), ((1024, 8, 8), .1),
                                   ((8, 1024, 8), .3), ((8, 8, 1024), 1.), ((150, 96, 100), 3.)])
def test_sweeps_at_segment_edges(gpe_lib, oracle_mod, mode, prec, n, dtf):
    s, o, psi = pair(gpe_lib, oracle_mod, mode, prec, n, dtf)
    for name in ("calclux", "calcluy", "calcluz"):
        s.set_psi(psi)
        o.set_psi(psi)
        getattr(s, name)()
        getattr(o, name)()
        assert rel(s.get_psi(), o.get_psi()) <= TOL[prec], name
    s.close()
    o.close()


# Time steps whose carries reach all segments of a line (D = P): c = dt / (2 dx^2)
# is 100.  The FP64 bar stands.  In FP32 the right-hand side psi + A t has terms of
# 4c times psi, each rounded at 2^-24.  In imaginary time the inverse that follows
# is bounded by 1; in real time each of the two recurrences passes such a rounding
# on over about sqrt(c) points before it has decayed.
@pytest.mark.parametrize("mode,prec,tol", [(0, 0, 1e-12), (1, 0, 1e-12), (0, 1, 2 ** -24 * 400), (1, 1, 2 ** -24 * 400 * 2 * 10)])
@pytest.mark.parametrize("n", [(96, 128, 80), (250, 36, 64), (18, 300, 24)])
def test_sweeps_at_large_time_steps(gpe_lib, oracle_mod, mode, prec, tol, n):
    s, o, psi = pair(gpe_lib, oracle_mod, mode, prec, n, 200.)
    for name in ("calclux", "calcluy", "calcluz"):
        s.set_psi(psi)
        o.set_psi(psi)
        getattr(s, name)()
        getattr(o, name)()
        assert rel(s.get_psi(), o.get_psi()) <= tol, name
    s.close()
    o.close()


@pytest.mark.parametrize("prec,tw,n", [(0, 4, (18, 10, 48)), (1, 4, (18, 10, 48)), (0, 2, (10, 18, 12)),
                                       (1, 8, (20, 12, 20))])
def test_narrow_tiles_keep_copies_aligned(gpe_lib, oracle_mod, prec, tw, n):
    """Tiles whose bytes are no multiple of 128: the phi tile behind the psi
    tile starts on a 128-byte boundary all the same."""
    s, o, psi = pair(gpe_lib, oracle_mod, 0, prec, n)
    t = gpe_lib.Tuning()
    t.sweep_tw[0] = t.sweep_tw[1] = t.sweep_tw[2] = tw
    s.set_tuning(t)
    s.calcnorm(True)
    o.calcnorm(True)
    s.run(2, 20., 5.)
    o.run(2, 20., 5.)
    assert rel(s.get_psi(), o.get_psi()) <= TOL[prec]
    s.close()
    o.close()


# exponents beyond each series' range: the per-point fallback of calcnu
@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("g", [1., 60., 2000.])
def test_calcnu_exponent_ranges(gpe_lib, oracle_mod, mode, prec, g):
    s, o, _ = pair(gpe_lib, oracle_mod, mode, prec, (30, 24, 20), 0.3)
    s.run(1, g, 0.)
    o.run(1, g, 0.)
    a, b = s.get_psi(), o.get_psi()
    # mixed precision in real time: the FP32 phase itself is rounded, to 2^-24
    # of its largest value, dt (V + g |psi|^2) <= 0.3 dx^2 (60 + 40 g)
    tol = max(TOL[prec], 2 ** -23 * 0.02 * (60. + 40. * g)) if prec and mode else TOL[prec]
    if prec and not mode:
        tol = max(tol, 2 ** -22 * 0.02 * 40. * g)
    assert rel(a, b) <= tol
    s.close()
    o.close()


# lengths with compile-time passes (24 ... 512 and half lengths) and without,
# odd half lengths, partial row tiles, the longest lines
@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("n", [(24, 32, 48), (48, 64, 96), (96, 24, 64), (128, 8, 128), (8, 256, 192), (512, 10, 16),
                               (10, 512, 512), (1024, 8, 20), (8, 1024, 24), (10, 8, 1024), (30, 50, 60), (90, 18, 36)])
def test_convolution_lengths(gpe_lib, oracle_mod, mode, prec, n):
    s, o, _ = pair(gpe_lib, oracle_mod, mode, prec, n)
    s.calcpsidd2()
    o.calcpsidd2()
    assert rel(s.get_phi(), o.get_phi()) <= TOL[prec]  # boundary planes included
    s.close()
    o.close()


@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("n", [(8, 8, 8), (20, 18, 36), (10, 36, 100), (48, 50, 32)])
def test_observables_at_tile_edges(gpe_lib, oracle_mod, mode, prec, n):
    s, o, _ = pair(gpe_lib, oracle_mod, mode, prec, n)
    assert s.calcnorm(False) == pytest.approx(o.calcnorm(False), rel=TOL[prec])
    assert s.calcmuen(30., 8.) == pytest.approx(o.calcmuen(30., 8.), rel=TOL[prec])
    assert np.allclose(s.calcrms(), o.calcrms(), rtol=TOL[prec], atol=0)
    for k in ("1d_z", "2d_xy"):
        assert rel(s.density(k), o.density(k)) <= TOL[prec], k
    s.close()
    o.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [(8, 8, 8), (10, 12, 20), (64, 40, 48)])
def test_mixed_psi_round_trip_is_exact(gpe_lib, mode, n):
    """psi of a mixed-precision handle is the caller's FP64 psi rounded once to
    FP32, in pieces of the spectrum buffer."""
    s = gpe_lib.Solver(gpe_lib.make_params(mode, *n, .25, .25, .25, .006, 1., 1., 1., 1., precision=1))
    r = np.random.default_rng(3)
    psi = r.standard_normal(n) + (1j * r.standard_normal(n) if mode else 0.)
    s.set_psi(psi)
    assert np.array_equal(s.get_psi(), psi.astype(np.complex64 if mode else np.float32))
    s.close()


# Lengths that have a compiled pass for one solve only: each of them along x, y
# and z (as a half length), against the oracle and against the run-time passes,
# which a largest radix of its own selects.
XY_LENGTHS = (16, 18, 20, 30, 36, 40, 50, 54, 60, 72, 80, 90, 100, 108, 120, 144, 150, 160, 162, 180, 192, 200, 216,
              240, 250, 288, 300, 320, 324, 360, 384, 400)
Z_HALVES = (8, 9, 10, 12, 15, 16, 18, 20, 25, 27, 30, 36, 40, 45, 50, 54, 60, 72, 75, 80, 81, 90, 100, 108, 120, 125,
            135, 144, 150, 160, 162, 180, 192, 200)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("axis,n", [(0, n) for n in XY_LENGTHS] + [(1, n) for n in XY_LENGTHS] +
                         [(2, 2 * h) for h in Z_HALVES])
def test_convolution_compiled_lengths(gpe_lib, oracle_mod, prec, axis, n):
    if prec and axis == 2 and n % 4:
        pytest.skip("mixed precision takes rows of a multiple of 4 points")
    shape = [10, 12, 8]
    shape[axis] = n
    s, o, psi = pair(gpe_lib, oracle_mod, 0, prec, tuple(shape))
    s.calcpsidd2()
    o.calcpsidd2()
    phi = s.get_phi()
    assert rel(phi, o.get_phi()) <= TOL[prec]
    t = gpe_lib.Tuning()
    t.fft_max_radix = 4
    s.set_tuning(t)
    s.set_psi(psi)
    s.calcpsidd2()
    assert rel(phi, s.get_phi()) <= TOL[prec]
    s.close()
    o.close()


# The forward z pass over complex rows: kernels of its own, with other row strides.
@pytest.mark.parametrize("prec,n", [(p, 2 * h) for p in (0, 1) for h in Z_HALVES if not (p and h % 2)])
def test_convolution_compiled_lengths_of_complex_rows(gpe_lib, oracle_mod, prec, n):
    s, o, psi = pair(gpe_lib, oracle_mod, 1, prec, (10, 12, n))
    s.calcpsidd2()
    o.calcpsidd2()
    phi = s.get_phi()
    assert rel(phi, o.get_phi()) <= TOL[prec]
    t = gpe_lib.Tuning()
    t.fft_max_radix = 4
    s.set_tuning(t)
    s.set_psi(psi)
    s.calcpsidd2()
    assert rel(phi, s.get_phi()) <= TOL[prec]
    s.close()
    o.close()


# A batch runs its own kernels on every length: the common ones compiled, the
# others at run time, on registers and points per thread that depend on which of
# the two its other members have.  Each instance is its solo run bit for bit.
@pytest.mark.parametrize("mode,prec", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("others", [(), ((64, 64, 64),), ((128, 48, 96), (24, 256, 32))])
def test_batch_lengths_bitwise(gpe_lib, mode, prec, others):
    gpe = gpe_lib
    shapes = list(others)
    for axis, lengths in enumerate((XY_LENGTHS + (270, 432, 640), XY_LENGTHS + (270, 486, 720),
                                    tuple(2 * h for h in Z_HALVES) + (432, 640))):
        for n in lengths:
            shape = [10, 12, 8]
            shape[axis] = n
            if not (prec and shape[2] % 4):
                shapes.append(tuple(shape))
    dx = 0.25
    ps = [gpe.make_params(mode, *n, dx, 1.1 * dx, 0.9 * dx, 0.1 * dx * dx, 0.5, 1.0, 1.5, 0.5 * min(n) * dx, precision=prec)
          for n in shapes]
    r = np.random.default_rng(7)
    psi = [r.standard_normal(n) * (0.3 + (0.2j if mode else 0.)) for n in shapes]
    g = [float(v) for v in r.uniform(1., 20., len(ps))]
    b = gpe.Batch(ps, g, [0.2 * v for v in g])
    for i, f in enumerate(psi):
        b.solver(i).set_psi(f)
    b.run(2)
    bad = []
    for i, p in enumerate(ps):
        with gpe.Solver(p) as s:
            s.set_tuning(b.solver(i).get_tuning())
            s.set_psi(psi[i])
            s.run(2, g[i], 0.2 * g[i])
            if not np.array_equal(s.get_psi(), b.solver(i).get_psi()):
                bad.append(shapes[i])
    b.close()
    assert not bad, bad

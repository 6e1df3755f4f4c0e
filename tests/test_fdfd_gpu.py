"""orf.fdfd2D on the device (opticrcwafdtd_b200/fdfd.py, csrc/fdfd.cu) against
the FDFD oracle, on the reference's own physics checks
(tests/TestInverseDesign.m:12-33), and its adjoint gradient."""
import threading

import numpy as np
import pytest

import opticrcwafdtd_b200 as orf
from oracle.fdfd import fdfd2D as oracle_fdfd2D
from tests import fdfd_cases

pytestmark = pytest.mark.gpu

# Both sides are direct solves with partial pivoting of the same FP64
# matrix; they differ by rounding amplified by the operator's conditioning.
TOL = 1e-9


def rel(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


@pytest.mark.parametrize("nx,nz,lossy", [(60, 40, True), (45, 70, False), (300, 150, True), (170, 400, True),
                                         (420, 300, False)])
def test_fdfd_matches_oracle(nx, nz, lossy):
    # blocks of 40 .. 300 points: every cluster shape of the solver, both orientations
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(nx, nz, nx + nz, lossy)
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    r = oracle_fdfd2D(x, z, eps, lam, J, Npml=npml)
    assert rel(o.E, r.E) <= TOL
    assert rel(o.adjoint(g), r.adjoint(g)) <= TOL
    J2 = np.roll(J, 5, axis=0) * 1j
    assert rel(o.solve(J2), r.solve(J2)) <= TOL
    info = o.info()
    assert info["block"] == min(nx, nz) and info["blocks"] == max(nx, nz)
    o.close()


def test_fdfd_straight_guide_is_exact():
    x, z, epsr, lam, J, m, win = fdfd_cases.straight_guide()
    o = orf.fdfd2D(x, z, epsr, lam, J)
    fdfd_cases.check_straight_guide(o, x, z, m, win)
    r = oracle_fdfd2D(x, z, epsr, lam, J)
    assert rel(o.E, r.E) <= TOL


def test_fdfd_adjoint_gradient_matches_finite_differences():
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(50, 36, 8)
    ctx = orf.Context(0)
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml, ctx=ctx)
    grad = -o.k0 ** 2 * o.adjoint(g) * o.E
    h = 1e-6
    for (i, k) in ((20, 18), (40, 6), (5, 30)):
        ep, em = eps.copy(), eps.copy()
        ep[i, k] += h
        em[i, k] -= h
        cp = np.sum(g * orf.fdfd2D(x, z, ep, lam, J, Npml=npml, ctx=ctx).E)
        cm = np.sum(g * orf.fdfd2D(x, z, em, lam, J, Npml=npml, ctx=ctx).E)
        assert abs((cp - cm) / (2 * h) - grad[i, k]) <= 1e-6 * max(1.0, abs(grad[i, k]))
    o.close()
    ctx.close()


def test_fdfd_rejects_a_block_above_the_limit():
    x = np.arange(400) * 0.02
    with pytest.raises(orf.OrfError) as ei:
        orf.fdfd2D(x, x, np.ones((400, 400)), 1.55, np.zeros((400, 400)))
    assert ei.value.identifier == "orf:tooLarge"


@pytest.mark.parametrize("nx,nz", [(3, 5), (9, 3), (64, 90), (80, 65), (128, 140), (131, 129), (256, 260), (258, 257),
                                   (384, 386)])
def test_fdfd_block_shapes(nx, nz):
    """Blocks at the edges of the cluster shapes (up to 64, 128, 256 and 384
    points), grids of one segment and of many, and the trailing rows and
    panels that a cluster's CTAs share unevenly."""
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(nx, nz, 3 * nx + nz, True, npml=(min(8, (nx - 1) // 2),
                                                                                        min(6, (nz - 1) // 2)))
    J[nx // 3, nz // 4:3 * nz // 4 + 1] = 1.0 + 0.3j   # (a line current on the smallest grids too)
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    r = oracle_fdfd2D(x, z, eps, lam, J, Npml=npml)
    assert rel(o.E, r.E) <= TOL
    assert rel(o.adjoint(g), r.adjoint(g)) <= TOL
    o.close()


def test_fdfd_segment_in_resonance():
    """A closed lossless cavity with five segments of five lines that, cut off
    by themselves, are exactly in resonance (k0^2 eps is an eigenvalue of the
    5 x 6-point Laplacian: condition number 1e17); the first and the last five
    lines hold other materials, so neither the whole grid (1.9e2) nor what the
    elimination from the first line meets (2.7e3) is.  The factorisation has
    to notice and go on as one segment.  41 lines are cut into seven segments
    of five and six separators."""
    nx, nz, d, lam = 41, 6, 0.03, 1.3
    k0 = 2 * np.pi / lam
    ev = 4 / d ** 2 * (np.sin(np.pi / (2 * 6)) ** 2 + np.sin(np.pi / (2 * 7)) ** 2)
    eps = np.full((nx, nz), ev / k0 ** 2)
    eps[:5] *= 1.3
    eps[36:] *= 1.5
    rng = np.random.default_rng(5)
    J = rng.standard_normal((nx, nz)) + 1j * rng.standard_normal((nx, nz))
    x, z = np.arange(nx) * d, np.arange(nz) * d
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=(0, 0))
    r = oracle_fdfd2D(x, z, eps, lam, J, Npml=(0, 0))
    assert rel(o.E, r.E) <= TOL
    assert rel(o.adjoint(J), r.adjoint(J)) <= TOL
    o.close()


@pytest.mark.parametrize("nx,nz", [(12, 9), (170, 60), (90, 240)])
def test_fdfd_refuses_a_permittivity_that_is_not_a_number(nx, nz):
    """One NaN cell makes every pivot row NaN sooner or later: refused as a
    singular operator, as one segment (12 x 9) and as many."""
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(nx, nz, 5, True, npml=(3, 3))
    eps[nx // 2, nz // 3] = np.nan
    with pytest.raises(orf.OrfError) as ei:
        orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    assert ei.value.identifier == "orf:invalidInput"


@pytest.mark.parametrize("nx,nz,cut", [(3, 5, False), (8, 6, False), (64, 90, True), (131, 129, True), (258, 257, True)])
def test_fdfd_reports_its_segments(nx, nz, cut):
    """The factors of an ordinary grid are those planned; grids of a hundred
    lines are cut, the smallest are not."""
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(nx, nz, 2, True, npml=(min(8, (nx - 1) // 2),
                                                                                min(6, (nz - 1) // 2)))
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    info = o.info()
    o.close()
    assert info["segments"] == info["planned_segments"]
    assert (info["segments"] > 1) == cut


@pytest.mark.parametrize("nb,planned", [(9, 2), (14, 3), (35, 6), (41, 7), (60, 9)])
def test_fdfd_odd_and_even_separator_counts(nb, planned):
    """Two to nine segments (one to eight separators, met in the middle from
    both ends): odd and even counts, against the oracle."""
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(nb, 7, nb, True, npml=(2, 2))
    J[nb // 3, 1:6] = 1.0 + 0.3j
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    r = oracle_fdfd2D(x, z, eps, lam, J, Npml=npml)
    info = o.info()
    assert info["planned_segments"] == planned and info["segments"] == planned
    assert rel(o.E, r.E) <= TOL
    assert rel(o.adjoint(g), r.adjoint(g)) <= TOL
    o.close()


def test_fdfd_segment_in_resonance_falls_back_to_one():
    """The cavity of test_fdfd_segment_in_resonance: planned as seven
    segments, five of them singular by themselves, factored as one."""
    nx, nz, d, lam = 41, 6, 0.03, 1.3
    ev = 4 / d ** 2 * (np.sin(np.pi / (2 * 6)) ** 2 + np.sin(np.pi / (2 * 7)) ** 2)
    eps = np.full((nx, nz), ev / (2 * np.pi / lam) ** 2)
    eps[:5] *= 1.3
    eps[36:] *= 1.5
    o = orf.fdfd2D(np.arange(nx) * d, np.arange(nz) * d, eps, lam, np.ones((nx, nz)), Npml=(0, 0))
    info = o.info()
    o.close()
    assert info["planned_segments"] == 7 and info["segments"] == 1


def test_fdfd_factorisations_on_several_threads():
    """Blocks of 150 and of 250 points are factored by one kernel with
    different shared memory sizes: side by side on two threads, each with its
    own context, neither changes what the other may launch."""
    probs = [fdfd_cases.random_problem(nx, nz, nx, True) for nx, nz in ((160, 150), (260, 250))]
    first, got, errs = [], [[], []], []

    def work(q, n):
        x, z, eps, lam, J, g, npml = probs[q]
        ctx = orf.Context(0)
        try:
            for _ in range(n):
                o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml, ctx=ctx)
                got[q].append((o.info()["segments"], o.E))
                o.close()
        except Exception as e:   # noqa: BLE001 (a thread's failure is the test's)
            errs.append(e)
        ctx.close()

    for q in (0, 1):   # alone
        work(q, 1)
        first.append(got[q].pop())
    th = [threading.Thread(target=work, args=(0, 150)), threading.Thread(target=work, args=(1, 60))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errs, errs
    for q in (0, 1):
        assert first[q][0] > 1
        assert all(s == first[q][0] and np.array_equal(E, first[q][1]) for s, E in got[q])


@pytest.mark.parametrize("nx,nz", [(120, 40), (33, 150)])
@pytest.mark.parametrize("power", [-1000, -660, 660, 960])
def test_fdfd_solution_scales_with_its_source(nx, nz, power):
    """A source times a power of two gives the field times that power, to the
    bit: the residual check and its refinement see the same numbers at
    1e-300 as at 1."""
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(nx, nz, 3, True)
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    assert o.info()["segments"] > 1
    s = 2.0 ** power
    assert np.array_equal(o.solve(J * s), np.ldexp(o.E.real, power) + 1j * np.ldexp(o.E.imag, power))
    a = o.adjoint(g)
    assert np.array_equal(o.adjoint(g * s), np.ldexp(a.real, power) + 1j * np.ldexp(a.imag, power))
    r = oracle_fdfd2D(x, z, eps, lam, J, Npml=npml)
    assert rel(o.E, r.E) <= TOL
    o.close()


@pytest.mark.parametrize("detuning", [0.0, 1e-8, 1e-5, 1e-4, 5e-4, 1e-3, 3e-3, 1e-2])
def test_fdfd_segments_near_resonance(detuning):
    """The cavity of test_fdfd_segment_in_resonance moved off its segments'
    resonance by a little: trial residuals from far above what is refused to
    that of an ordinary operator.  Sources all over, on one cell and in the
    shape of a segment's mode: the residual is that of a stable solve however
    many segments the factors keep, and the field and adjoint the oracle's."""
    nx, nz, d, lam = 41, 6, 0.03, 1.3
    ev = 4 / d ** 2 * (np.sin(np.pi / (2 * 6)) ** 2 + np.sin(np.pi / (2 * 7)) ** 2)
    eps = np.full((nx, nz), ev * (1 + detuning) / (2 * np.pi / lam) ** 2)
    eps[:5] *= 1.3
    eps[36:] *= 1.5
    x, z = np.arange(nx) * d, np.arange(nz) * d
    rng = np.random.default_rng(6)
    every = rng.standard_normal((nx, nz)) + 1j * rng.standard_normal((nx, nz))
    cell, mode = np.zeros((2, nx, nz))
    cell[14, 2] = 1.0
    mode[12:17] = np.outer(np.sin(np.pi * np.arange(1, 6) / 6), np.sin(np.pi * np.arange(1, 7) / 7))
    o = orf.fdfd2D(x, z, eps, lam, every, Npml=(0, 0))
    r = oracle_fdfd2D(x, z, eps, lam, every, Npml=(0, 0))
    assert o.info()["planned_segments"] == 7
    for J in (every, cell, mode):
        for a, b in ((o.solve, r.solve), (o.adjoint, r.adjoint)):
            assert rel(a(J), b(J)) <= TOL
            assert 0.0 <= o.info()["residual"] <= 1e-15
    o.close()


def test_fdfd_source_that_has_no_residual():
    """A source with a NaN or an infinity, and one of zeros, are solved as they
    are: the factors stay, and the next solve is the first one's to the bit."""
    x, z, eps, lam, J, g, npml = fdfd_cases.random_problem(120, 40, 4, True)
    o = orf.fdfd2D(x, z, eps, lam, J, Npml=npml)
    planned = o.info()["planned_segments"]
    assert planned > 1
    for bad in (np.nan, np.inf):
        Jb = J.copy()
        Jb[60, 20] = bad
        assert not np.all(np.isfinite(o.solve(Jb)))
        assert np.isnan(o.info()["residual"])
    assert np.all(o.solve(0 * J) == 0) and np.all(o.adjoint(0 * g) == 0)
    assert o.info()["residual"] == 0.0
    assert np.array_equal(o.solve(J), o.E)
    assert o.info()["segments"] == planned and 0.0 < o.info()["residual"] <= 1e-15
    o.close()

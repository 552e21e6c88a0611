"""The predictor's line solvers against the CPU oracle, where a wrong end, a
wrong solver or a wrong order of the boundary fills shows: symmetry walls with
a normal velocity, couplings on both sides of each dispatch line, no diffusion
at all, threads with lines of different lengths.

The oracle eliminates the same matrices; both are stable, so the fields agree to
a few rounding errors of their largest value: 1e-13 of it.
"""
import threading
from fractions import Fraction

import numpy as np
import pytest

import pyoracle as po
import solver_b200 as sb
from conftest import to_gpu_bc, to_gpu_grid

pytestmark = pytest.mark.gpu


def _compare(oracle, g, bc, alpha, rhs):
    with sb.Context(to_gpu_grid(g), to_gpu_bc(bc)) as ctx:
        got, lines = ctx.solve_predictor_adi(rhs, alpha)
    exp, lines_ref = oracle.predictor_adi(g, bc, alpha, *rhs)
    assert lines == lines_ref
    for a, b in zip(got, exp):
        assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))


def _rhs(g, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal(po.shape(g, c)) for c in "uvw"]


@pytest.mark.parametrize("alpha", [0.002, 0.1, 0.3, 40.0])
@pytest.mark.parametrize("shape", [(9, 12, 10), (40, 9, 33)], ids=lambda s: "x".join(map(str, s)))
def test_symmetry_wall_with_normal_velocity(oracle, shape, alpha):
    """The sweep along a symmetry wall's own axis takes the face's stored normal
    velocity like every fixed wall (the face itself is then set to zero)."""
    g = po.Grid(*shape, 0.5, 0.6, 0.55)
    bc = po.bc_from([po.SYMMETRY, po.SYMMETRY, po.NO_SLIP_WALL, po.SYMMETRY, po.SYMMETRY, po.NO_SLIP_WALL],
                    [(0.7, 0.1, 0.2), (-0.3, 0.0, 0.0), None, (0.2, 0.4, 0.1), (0.0, 0.0, 0.9), None])
    _compare(oracle, g, bc, alpha, _rhs(g, 3))


@pytest.mark.parametrize("alpha", [3e2, 1e14, 1e15, 1e16, 1e17, 1e19, 1e33])
def test_couplings_without_a_decay_length(oracle, alpha):
    """Couplings whose decay length is thousands of cells, exceeds every int or
    does not exist (lambda rounds to 1) take the eliminations.  Fixed walls: the
    matrix tends to the second difference, of condition 4 (n / pi)^2 = 650 for
    the longest line (40), so the fields agree to 650 x 8 roundings: 1e-12."""
    g = po.Grid(40, 12, 33, 0.5, 0.6, 0.55)
    bc = po.bc_from([po.NO_SLIP_WALL, po.PRESCRIBED_VELOCITY] * 3,
                    [None, (0.4, 0.2, -0.3), None, (0.7, -0.5, 0.1), None, (0.3, 0.2, 0.6)])
    rhs = _rhs(g, 4)
    with sb.Context(to_gpu_grid(g), to_gpu_bc(bc)) as ctx:
        got, lines = ctx.solve_predictor_adi(rhs, alpha)
    exp, lines_ref = oracle.predictor_adi(g, bc, alpha, *rhs)
    assert lines == lines_ref
    for a, b in zip(got, exp):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


@pytest.mark.parametrize("alpha", [0.001, 1.0])
def test_threads_with_lines_of_different_lengths(alpha):
    """Six contexts in six threads, half of them with lines that need far more
    shared memory than the others', solving and building plans at the same time: a
    launch must not depend on the sizes of another thread's."""
    failed = []

    def work(shape):
        try:
            g = sb.Grid(*shape, 0.1, 0.1, 0.1)
            rhs = [np.ones(g.shape(c)) for c in "uvw"]
            for _ in range(4):
                with sb.Context(g, [sb.PERIODIC] * 6) as ctx:
                    ctx.project_velocity(rhs, 0.01, 1.0, 5, 1e-6)
                    for _ in range(400):
                        out, _ = ctx.solve_predictor_adi(rhs, alpha)
                    for o in out:  # a constant is unchanged
                        assert np.max(np.abs(o[1:-1, 1:-1, 1:-1] - 1.0)) <= 1e-12
        except Exception as e:
            failed.append((shape, e))

    threads = [threading.Thread(target=work, args=(s,)) for s in ((1000, 2, 1), (16, 2, 1)) * 3]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("shape", [(9, 12, 10), (16, 8, 1), (1, 9, 7)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("types", ["walls", "open", "periodic"])
def test_no_diffusion_fills_the_boundaries_once(oracle, shape, types):
    """alpha = 0: no sweep, and the ghosts are filled from the faces as they were
    passed in, which only then are set (bitwise: nothing is computed but
    2 value - neighbour)."""
    g = po.Grid(*shape, 0.5, 0.6, 0.55)
    sets = {"walls": [po.NO_SLIP_WALL, po.PRESCRIBED_VELOCITY, po.SYMMETRY, po.PRESCRIBED_VELOCITY,
                      po.NO_SLIP_WALL, po.SYMMETRY],
            "open": [po.PRESCRIBED_VELOCITY, po.FIXED_PRESSURE, po.NO_SLIP_WALL, po.NO_SLIP_WALL,
                     po.PERIODIC, po.PERIODIC],
            "periodic": [po.PERIODIC] * 6}
    vel = [(0.25, 0.3, -0.2), (0.4, 0.2, -0.3), None, (0.7, -0.5, 0.1), None, None]
    bc = po.bc_from(sets[types], [None] * 6 if types == "periodic" else vel)
    rhs = _rhs(g, 5)
    with sb.Context(to_gpu_grid(g), to_gpu_bc(bc)) as ctx:
        got, _ = ctx.solve_predictor_adi(rhs, 0.0)
    exp, _ = oracle.predictor_adi(g, bc, 0.0, *rhs)
    for a, b in zip(got, exp):
        assert np.array_equal(a, b)


ENDS = {
    "periodic": ([po.PERIODIC] * 6, [None] * 6),
    "walls": ([po.NO_SLIP_WALL, po.PRESCRIBED_VELOCITY, po.SYMMETRY, po.PRESCRIBED_VELOCITY, po.NO_SLIP_WALL,
               po.SYMMETRY],
              [None, (0.4, 0.2, -0.3), (0.1, 0.6, 0.0), (0.7, -0.5, 0.1), None, (0.2, 0.0, -0.8)]),
    "open": ([po.PRESCRIBED_VELOCITY, po.FIXED_PRESSURE, po.FIXED_PRESSURE, po.NO_SLIP_WALL, po.PERIODIC,
              po.PERIODIC],
             [(1.0, 0.3, -0.2), None, None, None, None, None]),
}


# lines of one chunk (16 unknowns) and an unknown less or more, of two, and with
# 32, 16 and 8 lines to a block; rows on both sides of the lengths where 16 and
# 4 of them share one
@pytest.mark.parametrize("types", list(ENDS))
@pytest.mark.parametrize("shape", [(8, 15, 16), (17, 31, 8), (33, 9, 32), (16, 500, 3), (3, 520, 9), (5, 1030, 2),
                                   (1030, 16, 1), (700, 70, 70)],
                         ids=lambda s: "x".join(map(str, s)))
def test_chunks_of_a_line(oracle, shape, types):
    g = po.Grid(*shape, 0.5, 0.6, 0.55)
    bc = po.bc_from(*ENDS[types])
    for alpha in (1e-6, 0.05, 0.6):
        _compare(oracle, g, bc, alpha, _rhs(g, sum(shape)))


@pytest.mark.parametrize("types", ["periodic", "no_slip"])
def test_small_unknowns_keep_their_relative_accuracy(oracle, types):
    """The response to one large entry falls by many powers of ten along each
    axis; every one of its values agrees with the elimination's relatively.
    Either side multiplies one rounded factor per cell (both carry a few units
    of 1.1e-16 each over at most 90 + 70 + 50 cells: below 1e-13), and wall images
    of the other sign cancel less than two digits: 1e-11."""
    g = po.Grid(90, 70, 50, 0.5, 0.5, 0.5)
    bc = po.bc_from([po.PERIODIC] * 6 if types == "periodic" else [po.NO_SLIP_WALL] * 6)
    rhs = [np.zeros(po.shape(g, c)) for c in "uvw"]
    for r in rhs:
        r[20, 30, 40] = 1.0
    with sb.Context(to_gpu_grid(g), to_gpu_bc(bc)) as ctx:
        got, _ = ctx.solve_predictor_adi(rhs, 0.3)
    exp, _ = oracle.predictor_adi(g, bc, 0.3, *rhs)
    for a, b in zip(got, exp):
        a, b = po.active(a), po.active(b)
        assert np.min(np.abs(b[b != 0.0])) < 1e-25
        assert np.all(np.abs(a - b) <= 1e-11 * np.abs(b))


@pytest.mark.parametrize("beta", [2.45, 2.55, 30.0])
@pytest.mark.parametrize("types", ["walls", "periodic"])
@pytest.mark.parametrize("shape", [(200, 130, 1), (1000, 40, 1), (96, 70, 12), (128, 64, 10)],
                         ids=lambda s: "x".join(map(str, s)))
def test_both_sides_of_the_coupling_limit(oracle, shape, types, beta):
    """alpha / h^2 just below the chunked solver's limit (2.5) and above it, where
    lines of 64 to 1024 unknowns take the warp scan: wall lines whose length is not
    a multiple of 32 (199, 999, 95, 69 unknowns) padded to one, few long lines (2D)
    four to a block, periodic ones that do not divide one thread each.  The
    matrices' condition is at most 1 + 4 beta = 121: 1e-13 still holds."""
    g = po.Grid(*shape, 0.5, 0.5, 0.5)
    bc = po.bc_from(*ENDS[types])
    _compare(oracle, g, bc, beta * 0.25, _rhs(g, sum(shape)))


@pytest.mark.parametrize("beta", [0.001, 0.05, 0.13793428401297597, 0.3, 0.7, 2.2])
def test_sweeps_neither_damp_nor_feed_the_mean(beta):
    """The matrix's diagonal is 1 + 2 beta as rounded, so each sweep divides a
    periodic field's mean by its row's sum, 1 but for that rounding.  A constant of
    the solver that is rounded differently would move the mean the same way in every
    sweep, 1.1e-16 at a time: 7e-15 in 60.  What may remain is the rounding of the
    factor at the chunks' ends (1.1e-16 lambda / (1 - lambda) on one unknown in 16,
    at most 8e-18 of the mean) and the average of single roundings: 1e-17 a sweep."""
    h = 0.5
    g = po.Grid(24, 20, 28, h, h, h)
    bc = po.bc_from([po.PERIODIC] * 6)
    row = float(Fraction(1.0 + 2.0 * beta) - 2 * Fraction(beta) - 1)

    def means(fields):
        own = [tuple(slice(1, -2) if 2 - d == c else slice(1, -1) for d in range(3)) for c in range(3)]
        return [np.asarray(f[o], np.longdouble).mean() for f, o in zip(fields, own)]

    with sb.Context(to_gpu_grid(g), to_gpu_bc(bc)) as ctx:
        # alpha = 0 first: the duplicated faces are set to one value
        got, _ = ctx.solve_predictor_adi([1.0 + 0.5 * np.abs(r) for r in _rhs(g, 6)], 0.0)
        before = means(got)
        for _ in range(20):
            got, _ = ctx.solve_predictor_adi(got, beta * h * h)
    for m, b in zip(means(got), before):
        assert abs(float(m / b - 1) + 60 * row) <= 6e-16


@pytest.mark.parametrize("types", list(ENDS))
@pytest.mark.parametrize("shape", [(4095, 3, 1), (4097, 3, 2), (2, 2050, 3), (3, 8200, 1), (2, 16384, 1), (1, 16385, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_longest_lines(oracle, shape, types):
    """Rows of up to 4096 unknowns and columns of up to 16384 are solved in chunks
    (four rows, or as few as one column, to a block of 1024 threads), longer ones
    by one thread each."""
    g = po.Grid(*shape, 0.5, 0.6, 0.55)
    _compare(oracle, g, po.bc_from(*ENDS[types]), 0.2, _rhs(g, sum(shape)))

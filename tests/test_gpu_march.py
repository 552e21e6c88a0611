"""Pressure solves whose shapes sit at the edges of the marching kernels' tiles.

The V-cycle levels above 1024 cells and the CG updates run on tiles of row
patches (2 cells in FP64, 4 in FP32) that march k, with image cells outside
the domain; levels of at most 1024 cells are one matrix.  The shapes below
take rows that split into no whole patch, axes shorter than the halo, axes
that do not coarsen, one plane, one more cell than a tile and a finest level
that is itself the matrix, under every kind of boundary image.

The residual history of the first iterations is the reference's algorithm
iteration by iteration (a wrong image, weight or restriction changes it in the
first digits): it must agree to 1e-9 relative, far above the rounding of a few
V-cycles (about 1e-15 each) and far below any such error.  The solutions each
satisfy |b - A x| <= 1e-12 |b|, so they agree to 2e-12 times the condition
number of A (on the zero-mean subspace for singular problems).
"""
import numpy as np
import pytest

import pyoracle as po
from conftest import to_gpu_grid, to_gpu_pbc

pytestmark = pytest.mark.gpu

PER = [po.P_PERIODIC] * 6
NEU = [po.P_NEUMANN] * 6
MIX = [po.P_DIRICHLET, po.P_NEUMANN, po.P_PERIODIC, po.P_PERIODIC, po.P_NEUMANN, po.P_DIRICHLET]
DIR = [po.P_DIRICHLET] * 6

SHAPES = [
    (66, 28, 6),    # one more patch than a tile's 64 cells
    (130, 5, 3),    # odd rows, three planes
    (37, 20, 6),    # odd nx: no whole patches, x not coarsened
    (2, 36, 30),    # rows shorter than the halo
    (15, 18, 14),   # odd nx in a tile of one row of patches
    (20, 150, 2),   # two planes, many row tiles
    (70, 72, 1),    # one plane
    (257, 6, 1),    # one plane, odd nx above four tiles
    (32, 32, 2),    # level 1 is the matrix
    (16, 8, 8),     # the finest level is the matrix
]


def _condition(shape, h, types):
    """Largest over smallest non-zero eigenvalue of the separable operator."""
    lo, hi = [], []
    for a, n in enumerate(shape):
        m = np.zeros((n, n))
        for i in range(n):
            m[i, i] += 2.0
            for j, t in ((i - 1, types[2 * a]), (i + 1, types[2 * a + 1])):
                if 0 <= j < n:
                    m[i, j] -= 1.0
                elif t == po.P_PERIODIC:
                    m[i, j % n] -= 1.0
                else:
                    m[i, i] += 1.0 if t == po.P_DIRICHLET else -1.0
        e = np.sort(np.linalg.eigvalsh(m)) / h[a] ** 2
        lo.append(e)
        hi.append(e[-1])
    s = (lo[0][:, None, None] + lo[1][None, :, None] + lo[2][None, None, :]).ravel()
    return sum(hi) / np.min(s[s > 1e-9 * sum(hi)])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("types", [PER, NEU, MIX, DIR], ids=["periodic", "neumann", "mixed", "dirichlet"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_pressure_solve_at_tile_edges(oracle, shape, types, precision):
    import solver_b200 as sb
    h = (0.1, 0.12, 0.09)
    g = po.Grid(*shape, *h)
    rng = np.random.default_rng(sum(shape))
    rhs = rng.standard_normal(po.shape(g, "p"))
    pbc = po.pbc_from(types)
    ref = np.zeros(po.shape(g, "p"))
    dref, href = oracle.poisson_solve(g, pbc, 400, 1e-12, rhs, ref)
    assert dref.converged
    ctx = sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6,
                     precision=sb.OF_MIXED if precision == "mixed" else sb.OF_FP64)
    got, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(pbc), 2000, 1e-12)
    ctx.close()
    assert d["converged"] and d["relative_residual"] <= 1e-12
    if precision == "fp64":
        n = min(6, len(href), len(d["residual_history"]))
        np.testing.assert_allclose(d["residual_history"][:n], href[:n], rtol=1e-9, atol=1e-12 * href[0])
    a, b = po.active(got), po.active(ref)
    assert np.linalg.norm(a - b) <= 2e-12 * _condition(shape, h, types) * np.linalg.norm(b)


@pytest.mark.parametrize("amplitude", [1e-9, 1.0, 1e9])
@pytest.mark.parametrize("shape", [(30, 8, 5), (31, 9, 16), (32, 7, 17), (63, 17, 2), (5, 3, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_advection_at_tile_edges(oracle, shape, amplitude):
    """Tiles of 31 points along x (the 32nd lane evaluates the last face), rows
    of 8, chunks of planes with a carried face; amplitudes that take the
    limiter's quotient over many binades and its small-denominator branch.  Each
    flux is within a few rounding errors (the quotient within one ulp), so the
    term is within 1e-13 of its largest flux difference."""
    import solver_b200 as sb
    g = po.Grid(*shape, 0.3, 0.25, 0.4)
    rng = np.random.default_rng(sum(shape))
    vel = [amplitude * rng.standard_normal(po.shape(g, c)) for c in "uvw"]
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
        got = ctx.compute_advection_term(*vel)
    for a, b in zip(got, oracle.advection(g, *vel)):
        assert np.max(np.abs(po.active(a) - po.active(b))) <= 1e-13 * max(1e-300, np.max(np.abs(b)))


@pytest.mark.parametrize("alpha", [1e-6, 0.02, 0.3])
@pytest.mark.parametrize("types", ["periodic", "walls", "open"])
@pytest.mark.parametrize("shape", [(8, 9, 15), (16, 17, 33), (31, 32, 8), (100, 12, 40)],
                         ids=lambda s: "x".join(map(str, s)))
def test_adi_chunks_at_line_ends(oracle, shape, types, alpha):
    """Chunks of 16 unknowns whose reach (4 to 60 cells here) passes one or both
    ends of the line, several times over on the short ones: periodic images,
    wall reflections (with a moving lid and a wall-normal velocity) and
    fixed-pressure faces.  The images are exact up to the truncation at 2^-56
    and rounding: 1e-13 of the field's largest value."""
    import solver_b200 as sb
    from conftest import to_gpu_bc
    g = po.Grid(*shape, 0.5, 0.6, 0.55)
    sets = {"periodic": [po.PERIODIC] * 6,
            "walls": [po.NO_SLIP_WALL, po.PRESCRIBED_VELOCITY, po.SYMMETRY, po.PRESCRIBED_VELOCITY,
                      po.NO_SLIP_WALL, po.SYMMETRY],
            "open": [po.PRESCRIBED_VELOCITY, po.FIXED_PRESSURE, po.NO_SLIP_WALL, po.NO_SLIP_WALL,
                     po.PERIODIC, po.PERIODIC]}
    velocities = {"periodic": [None] * 6, "walls": [None, (0.4, 0.2, -0.3), None, (0.7, -0.5, 0.1), None, None],
                  "open": [(1.0, 0.3, -0.2), None, None, None, None, None]}
    bc = po.bc_from(sets[types], velocities[types])
    rng = np.random.default_rng(sum(shape))
    rhs = [rng.standard_normal(po.shape(g, c)) for c in "uvw"]
    with sb.Context(to_gpu_grid(g), to_gpu_bc(bc)) as ctx:
        got, lines = ctx.solve_predictor_adi(rhs, alpha)
    exp, lines_ref = oracle.predictor_adi(g, bc, alpha, *rhs)
    assert lines == lines_ref
    for a, b in zip(got, exp):
        assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("types", [PER, NEU], ids=["periodic", "neumann"])
@pytest.mark.parametrize("shape", [(48, 40, 32), (70, 72, 1)], ids=lambda s: "x".join(map(str, s)))
def test_solution_has_no_mean_whatever_the_guess(shape, types, precision):
    """Singular problems: the solution's mean is removed in every iteration, so a
    guess far from zero leaves none of its rounding (1e6 x 1e-16) behind: the mean
    of values of order one, rounded ones, is below 1e-15 of their size."""
    import solver_b200 as sb
    g = po.Grid(*shape, 0.02, 0.025, 0.03)
    rng = np.random.default_rng(sum(shape))
    rhs = rng.standard_normal(po.shape(g, "p"))
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6,
                    precision=sb.OF_MIXED if precision == "mixed" else sb.OF_FP64) as ctx:
        guess = 1e6 + rng.standard_normal(po.shape(g, "p"))
        got, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(po.pbc_from(types)), 400, 1e-10, pressure=guess)
    x = po.active(got)
    assert d["converged"] and d["iterations"] > 2
    assert abs(np.mean(x)) <= 1e-15 * np.sqrt(np.mean(x * x))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(2, 8192, 2), (4, 8192, 1), (3, 20480, 1), (8, 16384, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_narrow_and_long_planes(oracle, shape, precision):
    """Planes a few cells wide and many thousand long: a tile's rows are bounded
    by its shared memory, not by its threads.  The residuals of the first
    iterations as in test_pressure_solve_at_tile_edges."""
    import solver_b200 as sb
    g = po.Grid(*shape, 0.1, 0.12, 0.09)
    rng = np.random.default_rng(sum(shape))
    rhs = rng.standard_normal(po.shape(g, "p"))
    pbc = po.pbc_from(MIX)
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6,
                    precision=sb.OF_MIXED if precision == "mixed" else sb.OF_FP64) as ctx:
        if precision == "mixed":
            got, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(pbc), 4000, 1e-10)
            assert d["converged"] and d["relative_residual"] <= 1e-10
            return
        got, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(pbc), 5, 1e-12)
    ref = np.zeros(po.shape(g, "p"))
    _, href = oracle.poisson_solve(g, pbc, 5, 1e-12, rhs, ref)
    np.testing.assert_allclose(d["residual_history"], href, rtol=1e-9, atol=1e-12 * href[0])
    a, b = po.active(got), po.active(ref)
    assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(b))


def test_refused_plans_leave_no_device_memory():
    """A plan whose set-up fails (here: a coarsest level of 2500 unknowns) frees
    what it had allocated: thirty of 10 MB each would show."""
    import torch

    import solver_b200 as sb
    g = po.Grid(2, 20000, 4, 0.1, 0.1, 0.1)
    rhs = np.zeros(po.shape(g, "p"))
    pbc = to_gpu_pbc(po.pbc_from(PER))
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
        free = []
        for _ in range(30):
            with pytest.raises(ValueError, match="2500 unknowns"):
                ctx.solve_pressure_poisson(rhs, pbc, 5, 1e-6)
            free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 32 << 20


def _exact(shape, h, types, values, gradients, rhs):
    """The discrete solution of Lap p = rhs to well below FP64 rounding: the
    separable operator's eigenvectors, refined with residuals in extended
    precision."""
    mats, vecs, vals = [], [], []
    b = -np.asarray(rhs, np.longdouble)
    for a, n in enumerate(shape):
        m = np.zeros((n, n), np.longdouble)
        inv = np.longdouble(1.0) / (np.longdouble(h[a]) * np.longdouble(h[a]))
        for i in range(n):
            m[i, i] += 2
            for j, f in ((i - 1, 2 * a), (i + 1, 2 * a + 1)):
                if 0 <= j < n:
                    m[i, j] -= 1
                elif types[f] == po.P_PERIODIC:
                    m[i, j % n] -= 1
                elif types[f] == po.P_DIRICHLET:
                    m[i, i] += 1
                    face = [slice(None)] * 3
                    face[2 - a] = i
                    b[tuple(face)] += 2 * np.longdouble(values[f]) * inv
                else:
                    m[i, i] -= 1
                    face = [slice(None)] * 3
                    face[2 - a] = i
                    b[tuple(face)] += (1 if j == n else -1) * np.longdouble(gradients[f]) / np.longdouble(h[a])
        mats.append(m * inv)
        w, v = np.linalg.eigh(np.asarray(m, float))
        vals.append(w * float(inv))
        vecs.append(v)

    def apply(x, ms):
        return (np.einsum("ij,kli->klj", ms[0].T, x), np.einsum("ij,kil->kjl", ms[1].T, x),
                np.einsum("ij,ikl->jkl", ms[2].T, x))

    lam = vals[0][None, None, :] + vals[1][None, :, None] + vals[2][:, None, None]

    def solve(r):
        r = np.asarray(r, float)
        t = np.einsum("kji,il->kjl", np.einsum("kji,jl->kli", np.einsum("kji,kl->lji", r, vecs[2]), vecs[1]), vecs[0])
        t = t / lam
        return np.einsum("kji,li->kjl", np.einsum("kji,lj->kli", np.einsum("kji,lk->lji", t, vecs[2]), vecs[1]), vecs[0])

    x = np.zeros(b.shape, np.longdouble)
    for _ in range(4):
        x = x + solve(b - sum(apply(x, mats)))
    return x


@pytest.mark.parametrize("shape, h, types", [
    ((40, 63, 3), (0.32, 0.145, 0.077), [po.P_DIRICHLET, po.P_NEUMANN, po.P_PERIODIC, po.P_PERIODIC, po.P_NEUMANN,
                                         po.P_NEUMANN]),
    ((5, 2, 30), (0.15, 0.08, 1.57), [po.P_PERIODIC, po.P_PERIODIC, po.P_PERIODIC, po.P_PERIODIC, po.P_NEUMANN,
                                      po.P_DIRICHLET]),
    ((24, 20, 30), (0.2, 0.1, 0.5), [po.P_PERIODIC, po.P_PERIODIC, po.P_NEUMANN, po.P_NEUMANN, po.P_NEUMANN,
                                     po.P_DIRICHLET]),
    ((96, 40, 1), (0.5, 0.1, 1.0), [po.P_DIRICHLET, po.P_NEUMANN, po.P_NEUMANN, po.P_NEUMANN, po.P_NEUMANN,
                                    po.P_NEUMANN]),
], ids=["40x63x3", "5x2x30", "24x20x30", "96x40x1"])
def test_solution_is_as_accurate_as_the_reference_algorithm(oracle, shape, h, types):
    """A smooth solution many times larger than the residuals it is found from: the
    operator's terms are far larger than its values.  The error after a reduction of the
    residual by 1e-12 is the reference algorithm's (CPU oracle), give or take an
    iteration's progress: ten times it, or FP64 rounding of the solution."""
    import solver_b200 as sb
    g = po.Grid(*shape, *h)
    rng = np.random.default_rng(sum(shape))
    rhs = rng.standard_normal(po.shape(g, "p"))
    values = [-0.08, 0.0, 0.0, 0.0, 0.0, 1.3]
    gradients = [0.0, 0.005, 0.14, -0.7, 0.33, -0.68]
    gradients = [0.0 if t == po.P_PERIODIC else v for t, v in zip(types, gradients)]
    pbc = po.pbc_from(types, values, gradients)
    exact = _exact(shape, h, types, values, gradients, po.active(rhs))
    ref = np.zeros(po.shape(g, "p"))
    dref, _ = oracle.poisson_solve(g, pbc, 2000, 1e-12, rhs, ref)
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
        got, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(pbc), 4000, 1e-12)
    assert dref.converged and d["converged"]
    scale = float(np.sqrt(np.sum(exact * exact)))
    err, err_ref = (float(np.sqrt(np.sum((po.active(x) - exact) ** 2))) / scale for x in (got, ref))
    assert err <= 10 * max(err_ref, 1e-15)


def test_mixed_inner_solves_lose_no_iterations_to_the_operator(oracle):
    """Anisotropic cells, where the FP32 operator's terms are many digits above its
    values: cancelled digits would cost the inner solves iterations.  Restarting
    CG at a correction costs a part of the reference's count again (17 here), so
    1.6 times and a few is the limit."""
    import solver_b200 as sb
    shape, h = (5, 2, 30), (0.15, 0.08, 1.57)
    types = [po.P_PERIODIC] * 4 + [po.P_NEUMANN, po.P_DIRICHLET]
    g = po.Grid(*shape, *h)
    rng = np.random.default_rng(sum(shape))
    rhs, guess = rng.standard_normal(po.shape(g, "p")), rng.standard_normal(po.shape(g, "p"))
    pbc = po.pbc_from(types)
    dref, _ = oracle.poisson_solve(g, pbc, 1000, 1e-9, rhs, guess.copy())
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6, precision=sb.OF_MIXED) as ctx:
        _, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(pbc), 1000, 1e-9, pressure=guess.copy())
    assert dref.converged and d["converged"]
    assert d["iterations"] <= 1.6 * dref.iterations + 3


def test_constant_solves_its_own_problem():
    """The operator of a constant is its boundary terms to the last bit (spacings
    are powers of two, so these are exact): a guess that is the solution has no
    residual at all."""
    import solver_b200 as sb
    for shape in ((20, 18, 9), (33, 12, 1)):
        g = po.Grid(*shape, 0.25, 0.0625, 0.5)
        value = 1.0 / 3.0
        types = [po.P_DIRICHLET, po.P_DIRICHLET, po.P_PERIODIC, po.P_PERIODIC, po.P_NEUMANN, po.P_NEUMANN]
        pbc = po.pbc_from(types, [value, value, 0.0, 0.0, 0.0, 0.0])
        with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
            got, d = ctx.solve_pressure_poisson(np.zeros(po.shape(g, "p")), to_gpu_pbc(pbc), 50, 1e-12,
                                                pressure=np.full(po.shape(g, "p"), value))
        assert d["iterations"] == 0 and d["converged"]
        assert np.all(po.active(got) == value)


@pytest.mark.parametrize("shape", [(16, 12, 10), (32, 24, 1)], ids=lambda s: "x".join(map(str, s)))
def test_advection_passes_a_nan_on_like_the_reference(oracle, shape):
    """Every face value that a NaN enters is NaN, the ones it enters through the
    limiter's far neighbour included, and no other."""
    import solver_b200 as sb
    g = po.Grid(*shape, 0.1, 0.1, 0.1)
    rng = np.random.default_rng(8)
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
        for _ in range(12):
            vel = [rng.standard_normal(po.shape(g, c)) for c in "uvw"]
            f = vel[rng.integers(3)]
            f[tuple(int(rng.integers(1, n - 1)) for n in f.shape)] = np.nan
            got, exp = ctx.compute_advection_term(*vel), oracle.advection(g, *vel)
            for a, b in zip(got, exp):
                assert np.array_equal(np.isnan(po.active(a)), np.isnan(po.active(b)))


@pytest.mark.parametrize("shape", [(8, 8, 8), (20, 18, 6), (32, 24, 1)], ids=lambda s: "x".join(map(str, s)))
def test_alternating_boundary_conditions_and_precisions(shape):
    """One context that changes its problem from call to call (each change builds a
    plan, which takes over the last one's matrix memory where it fits) solves each
    as a fresh context does, bit for bit."""
    import solver_b200 as sb
    g = po.Grid(*shape, 0.1, 0.12, 0.09)
    rhs = np.random.default_rng(sum(shape)).standard_normal(po.shape(g, "p"))
    problems = [(t, p) for t in (PER, DIR, NEU, MIX) for p in (sb.OF_FP64, sb.OF_MIXED)]

    def solve(ctx, types, precision):
        ctx.set_precision(precision)
        x, d = ctx.solve_pressure_poisson(rhs, to_gpu_pbc(po.pbc_from(types)), 300, 1e-9)
        return np.array(x), d["iterations"]

    alone = []
    for types, precision in problems:
        with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
            alone.append(solve(ctx, types, precision))
    rng = np.random.default_rng(1)
    with sb.Context(to_gpu_grid(g), [sb.PERIODIC] * 6) as ctx:
        for k in rng.integers(0, len(problems), 40):
            x, it = solve(ctx, *problems[k])
            assert it == alone[k][1] and np.array_equal(x, alone[k][0])

"""The advection limiter's division: correctly rounded, on the host by itself and
on the GPU through the advection term."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotient_equals_the_division(tmp_path):
    exe = str(tmp_path / "quotient_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "quotient_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _values(kind, rng, shape):
    n = int(np.prod(shape))
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "binades":       # differences from below the limiter's 1e-14 up
        v = sign * rng.random(n) * 2.0 ** rng.integers(-48, -10, n)
    elif kind == "close":       # quotients next to num, delta or half of them
        v = 1e-6 * np.cumsum(1.0 + 1e-12 * rng.integers(-4, 5, n))
    elif kind == "patterns":    # fractions of all ones and powers of two
        v = sign * (2.0 - 2.0 ** -rng.integers(40, 53, n)) * 2.0 ** rng.integers(-40, -30, n)
    elif kind == "ones":        # quotients 2^k / d with a fraction of d of all ones
        v = np.zeros(shape)
        pairs = [(1.7071067811865472, 0.29289321881345254), (1.8660254037844384, 0.13397459621556138)]
        for j in range(shape[0]):
            for i in range(0, shape[1] - 3, 3):
                x, y = pairs[rng.integers(2)]
                assert x + y == 2.0 - 2.0 ** -52 and np.log2(x * y) in (-1.0, -2.0)
                v[j, i:i + 3] = np.array([-x, 0.0, y]) * 2.0 ** rng.integers(-40, -8) * rng.choice([-1.0, 1.0])
        return v
    elif kind == "tiny":        # products below the fast form's range
        v = np.where(rng.random(n) < 0.5, 1e-3 * rng.random(n), 1e-150 * rng.random(n))
    else:                       # products above it
        v = sign * rng.random(n) * 10.0 ** rng.integers(140, 153, n)
    return v.reshape(shape)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["binades", "close", "patterns", "ones", "tiny", "huge"])
def test_limiter_rounds_like_the_division(kind):
    """v varies along x only and u = 1, so the term is the difference of two
    limited face values, formed here operation by operation.  What the y faces
    add, a product and its own rounding error, is at most 2^-52 v^2 / dy: with
    dy = 1e160 far below the last bit of any face value."""
    import solver_b200 as sb
    nx = 96
    g = sb.Grid(nx, 16, 5, 1.0, 1e160, 1.0)
    rng = np.random.default_rng(len(kind))
    rows = _values(kind, rng, (16 + 3, nx + 2))
    rows[:] = rows[:1] if kind == "close" else rows
    results = []
    for row in rows[:6]:
        u, v, w = np.ones(g.shape("u")), np.empty(g.shape("v")), np.zeros(g.shape("w"))
        v[:] = row
        with sb.Context(g, [sb.PERIODIC] * 6) as ctx:
            got = ctx.compute_advection_term(u, v, w)[1]
        left, right, far = row[1:-1], row[2:], row[:-2]   # upper faces of points 1 .. nx, u > 0
        delta, num = right - left, left - far
        nd = num * delta
        on = (np.abs(delta) >= 1e-14) & (nd > 0.0)
        den = np.where(on, delta + num, 1.0)
        face = left + np.where(on, nd / den, 0.0)
        # the lower face of point 1 has no far value: first-order upwind
        exp = face - np.concatenate(([row[0]], face[:-1]))
        slack = 2.0 ** -52 * np.max(np.abs(row)) ** 2 / 1e160
        block = got[1:-1, 1:-1, 1:-1]
        assert block.shape[-1] == nx
        results.append(np.max(np.abs(block - exp)) <= slack)
    assert all(results)

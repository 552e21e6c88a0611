"""The coarse-level chain timing (of_profile_coarse_chain) on the GPU.

The bench times the V-cycle's coarse levels by replaying a CUDA graph of that
chain alone between steps.  Its contract: a positive time, the chain's launch
count, and no effect on later solves -- the replays rerun levels 1 ..
coarsest on the level-1 rhs of the last solve, and every value they write is
overwritten by the next solve's own V-cycles before it is read.  So a run
with replays between its steps must equal, bit for bit, the same run without
them.
"""
import numpy as np
import pytest

import solver_b200 as sb

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "adv_u", "adv_v", "adv_w", "p")


def _run(n, precision, profile):
    h = 2 * np.pi / n
    ctx = sb.Context(sb.Grid(n, n, n, h, h, h), [sb.PERIODIC] * 6, precision=precision)
    try:
        dt = 0.5 / (3.0 / h)
        ctx.tg_init(1.0 / 1600, dt, 1)
        prm = sb.step_params(1.0 / 1600, dt, 400, 1e-12)
        ctx.run_steps(prm, 2)
        chain = sb.profile_coarse_chain(ctx, 20) if profile else None
        m = ctx.run_steps(prm, 2)
        return ctx.download_state(), m, chain
    finally:
        ctx.close()


@pytest.mark.parametrize("precision", [sb.OF_FP64, sb.OF_MIXED])
def test_coarse_chain_replays_leave_the_run_bitwise_unchanged(precision):
    ref, m_ref, _ = _run(64, precision, False)
    out, m, (us, launches) = _run(64, precision, True)
    assert us > 0.0 and launches >= 1
    assert m["pressure_iterations"] == m_ref["pressure_iterations"]
    for f in FIELDS:
        assert np.array_equal(np.asarray(out[f]), np.asarray(ref[f])), f


@pytest.mark.parametrize("precision", [sb.OF_FP64, sb.OF_MIXED])
@pytest.mark.parametrize("shape", [(4, 4, 4), (8, 8, 8), (16, 8, 8), (32, 32, 1), (3, 3, 3)],
                         ids=lambda s: "x".join(map(str, s)))
def test_no_chain_below_a_dense_finest_level(shape, precision):
    """Grids of at most 1024 cells: the whole V-cycle is one matrix, nothing is
    launched below it.  The call says so, and neither the context nor the
    launch counters are left in a capture."""
    h = 2 * np.pi / max(shape)
    dt = 0.1 * h
    prm = sb.step_params(0.01, dt, 400, 1e-8)  # (4^3 breaks down at 1e-10: p.Ap < 1e-30)
    states, counts = [], []
    for profile in (False, True):
        with sb.Context(sb.Grid(*shape, h, h, h), [sb.PERIODIC] * 6, precision=precision) as ctx:
            ctx.tg_init(0.01, dt, 1)
            ctx.run_steps(prm, 1)
            if profile:
                assert sb.profile_coarse_chain(ctx, 3) == (0.0, 0)
            sb.profile_reset()
            ctx.run_steps(prm, 2)
            counts.append({k: v[0] for k, v in sb.profile_read().items()})
            states.append(ctx.download_state())
    assert counts[0] == counts[1] and sum(counts[0].values()) > 0
    for f in FIELDS:
        assert np.array_equal(np.asarray(states[0][f]), np.asarray(states[1][f])), f

"""Seam calls on pageable arrays large enough for the staged transfers.

Staged (pageable), plain (pinned) and contended (two threads at once, one of
which finds the staging slots taken) transfers move the same bytes: results
must be bitwise equal, and entries the reference leaves alone -- the ghosts of
the advection term and of the pressure fields -- must come back as passed in.
The sizes give fields below and above one slot (2 MiB) and storage rows that
straddle its chunks.
"""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

import solver_b200 as sb

pytestmark = pytest.mark.gpu

SIZES = [(28, 30, 24), (64, 62, 60), (96, 56, 144)]


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _calls(ctx, g, vel, wrap):
    rng = np.random.default_rng(7)
    adv = [wrap(rng.standard_normal(g.shape(c))) for c in "uvw"]
    before = [a.copy() for a in adv]
    ctx.compute_advection_term(*[wrap(v) for v in vel], out=adv)
    for a, b in zip(adv, before):
        ghost = np.ones(a.shape, bool)
        ghost[1:-1, 1:-1, 1:-1] = False
        assert np.array_equal(a[ghost], b[ghost])
        assert not np.array_equal(a[~ghost], b[~ghost])
    pred, lines = ctx.solve_predictor_adi([wrap(v) for v in vel], 0.002)
    phi, rhs = wrap(np.full(g.shape("p"), 0.25)), wrap(np.full(g.shape("p"), 0.5))
    out, _, _, _ = ctx.project_velocity([wrap(v) for v in vel], 0.01, 1.0, 60, 1e-6, pressure_correction=phi,
                                        pressure_rhs=rhs)
    for a, v in ((phi, 0.25), (rhs, 0.5)):
        ghost = np.ones(a.shape, bool)
        ghost[1:-1, 1:-1, 1:-1] = False
        assert np.all(a[ghost] == v)
    return [np.array(x) for x in adv + pred + out + [phi, rhs]]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_staged_transfers_equal_plain_ones(size):
    g = sb.Grid(*size, 0.1, 0.1, 0.1)
    bc = [sb.PERIODIC, sb.PERIODIC, sb.NO_SLIP_WALL, sb.NO_SLIP_WALL, sb.PERIODIC, sb.PERIODIC]
    rng = np.random.default_rng(1)
    vel = [rng.standard_normal(g.shape(c)) for c in "uvw"]
    with sb.Context(g, bc) as ctx:
        plain = _calls(ctx, g, vel, _pinned)
        staged = _calls(ctx, g, vel, np.array)
    for a, b in zip(plain, staged):
        assert np.array_equal(a, b)

    got = {}

    def work(k):
        with sb.Context(g, bc) as c:
            got[k] = _calls(c, g, vel, np.array)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        for a, b in zip(plain, got[k]):
            assert np.array_equal(a, b)


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import os, sys, time
sys.path.insert(0, {root!r})
import numpy as np
import solver_b200 as sb
g = sb.Grid(96, 96, 96, 0.1, 0.1, 0.1)
ctx = sb.Context(g, [sb.PERIODIC] * 6)
v = [np.ones(g.shape(c)) for c in "uvw"]
{body}
"""


def _run(body):
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", CHILD.format(root=ROOT, body=body)],
                       capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    return r.stdout.split()


@pytest.mark.parametrize("close", [False, True])
def test_forked_child_ends_normally(close):
    """The workers do not exist in a child of fork(): closing its copy of the
    context or leaving must not wait for them (nor crash)."""
    out = _run(f"""
for _ in range(3):  # 132 MB: the slots and workers exist
    ctx.compute_advection_term(*v)
time.sleep(0.05)
pid = os.fork()
if pid == 0:
    if {close}:
        ctx.close()
    sys.exit(0)
end = time.time() + 20
while time.time() < end:
    done, status = os.waitpid(pid, os.WNOHANG)
    if done:
        break
    time.sleep(0.02)
else:
    os.kill(pid, 9)
    status = "hangs"
ctx.compute_advection_term(*v)
ctx.close()
print(status)
""")
    assert out == ["0"]


@pytest.mark.parametrize("cpus", [1, 2])
def test_workers_fit_the_cpus_of_the_process(cpus):
    """A process held to few CPUs gets a worker less than it has CPUs, not one for
    every core of the machine."""
    if len(os.sched_getaffinity(0)) <= cpus:
        pytest.skip("too few CPUs to tell")
    out = _run(f"""
ctx.solve_predictor_adi([x[:] for x in v], 0.0)
os.sched_setaffinity(0, set(sorted(os.sched_getaffinity(0))[:{cpus}]))
before = len(os.listdir("/proc/self/task"))
for _ in range(4):
    ctx.compute_advection_term(*v)
print(len(os.listdir("/proc/self/task")) - before)
""")
    assert int(out[0]) <= cpus - 1


def test_slots_and_workers_only_where_they_pay():
    """A program that moves little is spared them; one that moves more gets them,
    loses them with its last context, and counts anew."""
    if len(os.sched_getaffinity(0)) < 2:
        pytest.skip("one CPU: no workers at all")
    out = _run("""
ctx.solve_predictor_adi([x[:] for x in v], 0.0)  # loads what is loaded once
ctx.close()
def workers(calls):
    c = sb.Context(g, [sb.PERIODIC] * 6)
    c.upload_state(*[np.zeros(g.shape(k)) for k in "uvwuvwp"], False)
    before = len(os.listdir("/proc/self/task"))
    for _ in range(calls):
        c.compute_advection_term(*v)
    n = len(os.listdir("/proc/self/task")) - before
    c.close()
    return n
print(workers(0), workers(4) > 0, workers(0))
""")
    assert out == ["0", "True", "0"]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_staged_transfers_equal_plain_ones_once_the_slots_exist(size):
    """As above for every size: another context has moved enough for the slots to
    be there from the first call on."""
    big = sb.Grid(96, 96, 96, 0.1, 0.1, 0.1)
    vel = [np.ones(big.shape(c)) for c in "uvw"]
    with sb.Context(big, [sb.PERIODIC] * 6) as holder:
        for _ in range(4):
            holder.compute_advection_term(*vel)
        test_staged_transfers_equal_plain_ones(size)

"""The work a program has this framework do, as cases that can be timed and compared.

Every case goes through the public entry points: ``solver_b200.Context`` (the
reference's four seam functions on host arrays, the step loop on a
device-resident state, the step of a host-resident state, the adjoint
gradient) and ``of_pressure_rhs_noalloc`` on device buffers.

``listed()`` are the cases of record, ``draw(rng)`` gives others of the same
ranges.  Inputs are made from a seed on the GPU: the Taylor-Green vortex, a
channel profile or a recirculating cavity flow, each with a smooth random
disturbance, on the grids and with the time step, viscosity and tolerance of
this repository's configurations and benchmark.  ``exact`` restates one call
in plain FP64 torch: the stencils as array slices, the line solves and the
pressure solve as dense (diagonalised) linear algebra, without an iteration.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import solver_b200 as sb
from solver_b200 import _capi

PER, WALL, LID, SYM = sb.PERIODIC, sb.NO_SLIP_WALL, sb.PRESCRIBED_VELOCITY, sb.SYMMETRY
LID_VELOCITY = (1.0, 0.0, 0.0)

# Velocity boundary sets by flow: the periodic box (its 2D form is one cell
# deep between symmetry planes), a channel with walls in y, the lid-driven
# cavity.
FLOWS = {
    "box": (PER, PER, PER, PER, PER, PER),
    "box2d": (PER, PER, PER, PER, SYM, SYM),
    "channel": (PER, PER, WALL, WALL, PER, PER),
    "cavity": (WALL, WALL, WALL, LID, SYM, SYM),
}
# Pressure boundary sets of a stand-alone solve; "outlet" fixes the pressure
# at x max, so that the problem has no null space.
PRESSURE = {
    "box": (sb.P_PERIODIC,) * 6,
    "channel": (sb.P_PERIODIC, sb.P_PERIODIC, sb.P_NEUMANN, sb.P_NEUMANN, sb.P_PERIODIC, sb.P_PERIODIC),
    "outlet": (sb.P_NEUMANN, sb.P_DIRICHLET, sb.P_NEUMANN, sb.P_NEUMANN, sb.P_NEUMANN, sb.P_NEUMANN),
}


def listed():
    return [
        # A program that owns all device memory forms the pressure right-hand
        # side of its own velocity buffers: the smallest device call there is.
        {"name": "rhs_64", "kind": "rhs", "nx": 64, "ny": 64, "nz": 64, "norms": True},
        # The reference tree with its advection seam replaced, on a small box
        # of odd proportions: host arrays in, host arrays out.
        {"name": "advect_48", "kind": "advect", "flow": "box", "nx": 48, "ny": 40, "nz": 36},
        # The implicit predictor of a channel of ragged size (line lengths that
        # are multiples of nothing), host arrays.
        {"name": "adi_channel", "kind": "adi", "flow": "channel", "nx": 130, "ny": 97, "nz": 51},
        # A stand-alone pressure solve with an outflow boundary, host arrays.
        {"name": "poisson_outlet", "kind": "poisson", "flow": "outlet", "nx": 96, "ny": 80, "nz": 72,
         "tol": 1e-10},
        # One projection of a predicted channel velocity, host arrays: the
        # largest of the reference's seams.
        {"name": "project_channel", "kind": "project", "flow": "channel", "nx": 128, "ny": 96, "nz": 64,
         "tol": 1e-10},
        # The shipped 2D Taylor-Green configuration: 128 x 128, 100 steps.
        {"name": "tg2d_128", "kind": "steps", "flow": "box2d", "nx": 128, "ny": 128, "nz": 1, "steps": 100,
         "nu": 0.01, "tol": 1e-12, "mixed": False},
        # The shipped 1024 x 1024 cavity configuration, a stretch of its march
        # to the steady state.
        {"name": "cavity_1024", "kind": "steps", "flow": "cavity", "nx": 1024, "ny": 1024, "nz": 1,
         "steps": 10, "nu": 0.01, "tol": 1e-8, "mixed": False},
        # A periodic box whose sides are no powers of two.
        {"name": "tg3d_odd", "kind": "steps", "flow": "box", "nx": 144, "ny": 80, "nz": 112, "steps": 5,
         "nu": 0.000625, "tol": 1e-12, "mixed": False},
        # The headline benchmark: Taylor-Green 256^3 at Re 1600, from one saved
        # state to the next.
        {"name": "tg3d_256", "kind": "steps", "flow": "box", "nx": 256, "ny": 256, "nz": 256, "steps": 8,
         "nu": 0.000625, "tol": 1e-12, "mixed": False},
        # The same with the pressure solve's V-cycle in FP32.
        {"name": "tg3d_256_mixed", "kind": "steps", "flow": "box", "nx": 256, "ny": 256, "nz": 256,
         "steps": 8, "nu": 0.000625, "tol": 1e-12, "mixed": True},
        # One step of a state that its owner keeps in (pinned) host memory: the
        # benchmark's end-to-end figure.
        {"name": "step_host_256", "kind": "step_host", "flow": "box", "nx": 256, "ny": 256, "nz": 256,
         "nu": 0.000625, "tol": 1e-12},
        # The gradient of a final-state misfit by the discrete adjoint, at the
        # size of the benchmark's adjoint check.
        {"name": "adjoint_128", "kind": "adjoint", "flow": "box", "nx": 128, "ny": 128, "nz": 128,
         "steps": 8, "every": 4, "nu": 0.01, "tol": 1e-12},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid_size(rng, lo, hi):
    """A size the multigrid hierarchy coarsens: an odd number up to 9 times a power of two."""
    sizes = sorted({m << k for m in (1, 3, 5, 7, 9) for k in range(1, 11) if lo <= m << k <= hi})
    want = math.log(lo) + rng.random() * (math.log(hi) - math.log(lo))
    return min(sizes, key=lambda n: abs(math.log(n) - want))


def draw(rng):
    kind = rng.choice(("rhs", "advect", "adi", "poisson", "project", "steps2d", "cavity", "steps3d", "steps3d",
                       "steps3d", "step_host", "adjoint"))
    if kind == "rhs":
        n = [_size(rng, 24, 288) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], norms=rng.random() < 0.5)
    if kind in ("advect", "adi"):
        n = [_size(rng, 20, 176) for _ in range(3)]
        return dict(kind=kind, flow=rng.choice(("box", "channel")), nx=n[0], ny=n[1], nz=n[2])
    if kind == "poisson":
        n = [_grid_size(rng, 16, 160) for _ in range(3)]
        return dict(kind=kind, flow=rng.choice(("box", "channel", "outlet")), nx=n[0], ny=n[1], nz=n[2],
                    tol=rng.choice((1e-8, 1e-10, 1e-12)))
    if kind == "project":
        n = [_grid_size(rng, 16, 160) for _ in range(3)]
        return dict(kind=kind, flow=rng.choice(("box", "channel")), nx=n[0], ny=n[1], nz=n[2], tol=1e-10)
    if kind == "steps2d":
        n = _grid_size(rng, 32, 512)
        return dict(kind="steps", flow="box2d", nx=n, ny=n, nz=1, steps=rng.randint(10, 40), nu=0.01, tol=1e-12,
                    mixed=False)
    if kind == "cavity":
        n = _grid_size(rng, 64, 896)
        return dict(kind="steps", flow="cavity", nx=n, ny=n, nz=1, steps=rng.randint(5, 20), nu=0.01, tol=1e-8,
                    mixed=False)
    if kind == "steps3d":
        n = [_grid_size(rng, 32, 224)] * 3
        if rng.random() < 0.5:  # a box of unequal sides
            n = [n[0], _grid_size(rng, max(16, n[0] * 2 // 3), n[0]), _grid_size(rng, max(16, n[0] // 2), n[0])]
        return dict(kind="steps", flow="box", nx=n[0], ny=n[1], nz=n[2], steps=rng.randint(2, 6),
                    nu=rng.choice((0.01, 0.000625)), tol=1e-12, mixed=rng.random() < 0.4)
    if kind == "step_host":
        n = _grid_size(rng, 96, 224)
        return dict(kind=kind, flow="box", nx=n, ny=n, nz=n, nu=0.000625, tol=1e-12)
    n = _grid_size(rng, 32, 112)
    return dict(kind="adjoint", flow="box", nx=n, ny=n, nz=n, steps=rng.randint(3, 8), every=rng.randint(1, 4),
                nu=0.01, tol=1e-12)


# ---------------------------------------------------------------------------
# geometry and inputs
# ---------------------------------------------------------------------------

def _grid(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case.get("flow") == "cavity":  # the unit square, one cell deep
        return sb.Grid(nx, ny, nz, 1.0 / nx, 1.0 / ny, 1.0)
    if nz == 1:
        return sb.Grid(nx, ny, nz, 2.0 * math.pi / nx, 2.0 * math.pi / ny, 1.0)
    if case["kind"] in ("steps", "step_host", "adjoint"):  # the Taylor-Green box
        return sb.Grid(nx, ny, nz, *(2.0 * math.pi / n for n in (nx, ny, nz)))
    h = 2.0 * math.pi / max(nx, ny, nz)  # cells of the same size in all directions
    return sb.Grid(nx, ny, nz, h, h, h)


def _dt(case):
    g = _grid(case)
    return 0.5 / (1.0 / g.dx + 1.0 / g.dy + (1.0 / g.dz if g.nz > 1 else 0.0))


def _bc(case):
    return sb.make_bc([(t, LID_VELOCITY) if t == LID else t for t in FLOWS[case["flow"]]])


def _params(case):
    variant = sb.OF_CORRECTION_CAVITY if case["flow"] == "cavity" else sb.OF_CORRECTION_TAYLOR_GREEN
    return sb.step_params(case["nu"], _dt(case), 400, case["tol"], variant=variant)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _coords(g, loc, dev):
    """Coordinates of a padded field's entries, (z, y, x), each broadcastable."""
    sz, sy, sx = g.shape(loc)
    out = []
    for n, h, c, shape in ((sz, g.dz, "w", (-1, 1, 1)), (sy, g.dy, "v", (1, -1, 1)), (sx, g.dx, "u", (1, 1, -1))):
        i = torch.arange(n, dtype=torch.float64, device=dev)
        out.append(((i - 1.0 if loc == c else i - 0.5) * h).reshape(shape))
    return out


def _noise(g, loc, rng, dev, amp, length, modes=5):
    """A smooth random field, periodic over `length` in each direction."""
    z, y, x = _coords(g, loc, dev)
    out = torch.zeros(g.shape(loc), dtype=torch.float64, device=dev)
    w = [2.0 * math.pi / l for l in length]
    for _ in range(modes):
        k = rng.integers(-4, 5, 3)
        a, ph = amp * rng.uniform(0.3, 1.0), rng.uniform(0.0, 2.0 * math.pi)
        out += a * torch.cos(k[0] * w[0] * x + k[1] * w[1] * y + (k[2] * w[2] * z if g.nz > 1 else 0.0 * z) + ph)
    return out


def _velocity(case, g, rng, dev):
    """Velocity (three padded fields) and total pressure of the case's flow."""
    length = (g.nx * g.dx, g.ny * g.dy, g.nz * g.dz)
    flow = case.get("flow", "box")
    swirl = rng.uniform(-0.05, 0.05, 3)
    fields = []
    for loc in "uvwp":
        z, y, x = _coords(g, loc, dev)
        zero = torch.zeros(g.shape(loc), dtype=torch.float64, device=dev)
        if flow == "cavity":
            # recirculation below the lid, psi = a sin^2(pi x) sin^2(m pi y) per mode m
            f, px = zero, math.pi * x
            for m, a in enumerate(swirl, 1):
                py = m * math.pi * y
                if loc == "u":
                    f = f + a * torch.sin(px) ** 2 * m * math.pi * torch.sin(2.0 * py)
                elif loc == "v":
                    f = f - a * math.pi * torch.sin(2.0 * px) * torch.sin(py) ** 2
            fields.append(f)
            continue
        if flow == "channel":
            eta = y * (1.0 / length[1])
            wall = 4.0 * eta * (1.0 - eta)
            f = wall * (1.0 if loc == "u" else 0.0) + _noise(g, loc, rng, dev, 0.05, length) * wall
            fields.append(f)
            continue
        sx, sy, sz = (2.0 * math.pi / l for l in length)
        x, y, z = x * sx, y * sy, z * sz
        zf = torch.cos(z) if g.nz > 1 else torch.ones_like(z)
        if loc == "u":
            f = torch.sin(x) * torch.cos(y) * zf
        elif loc == "v":
            f = -torch.cos(x) * torch.sin(y) * zf
        elif loc == "w":
            f = zero
        else:
            f = (torch.cos(2 * x) + torch.cos(2 * y)) * ((torch.cos(2 * z) + 2.0) / 16.0 if g.nz > 1
                                                        else torch.full_like(z, 0.25))
        amp = 0.0 if (g.nz == 1 and loc == "w") else 0.02
        fields.append(f + _noise(g, loc, rng, dev, amp, length) + zero)
    return fields


def _inputs(case, seed):
    """The seeded inputs as device tensors."""
    dev = _device()
    rng = np.random.default_rng(seed)
    g = _grid(case)
    if case["kind"] == "poisson":
        length = (g.nx * g.dx, g.ny * g.dy, g.nz * g.dz)
        rhs = _noise(g, "p", rng, dev, 1.0, length, modes=8)
        # the guess is what the last solve left: here nothing
        return {"rhs": rhs, "pressure": torch.zeros_like(rhs)}
    u, v, w, p = _velocity(case, g, rng, dev)
    out = {"u": u, "v": v, "w": w, "p": p}
    if case["kind"] == "adjoint":
        t = _velocity(case, g, rng, dev)
        out.update({"tu": t[0], "tv": t[1], "tw": t[2]})
    return out


def _host(t, pinned=False):
    if pinned and torch.cuda.is_available():
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
        h.copy_(t)
        return h.numpy()
    return t.cpu().numpy()


def _host_zeros(g, loc):
    return _host(torch.zeros(g.shape(loc), dtype=torch.float64), pinned=True)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    g = _grid(case)
    inp = _inputs(case, seed)
    kind = case["kind"]
    s = {"case": case, "grid": g}
    if kind == "rhs":
        s.update({k: inp[k].contiguous() for k in "uvw"})
        s["rhs"] = torch.zeros(g.shape("p"), dtype=torch.float64, device=inp["u"].device)
        s["norms"] = (ctypes.c_double * 2)()
        s["of_grid"] = _capi.OfGrid(g.nx, g.ny, g.nz, g.dx, g.dy, g.dz)
        s["dt"] = _dt(case)
        s["lib"] = _capi.load()
        return s
    if kind == "poisson":
        s["ctx"] = sb.Context(g, [PER] * 6)
        s["pbc"] = sb.make_pbc(PRESSURE[case["flow"]])
        s["rhs"] = _host(inp["rhs"])
        return s
    s["ctx"] = sb.Context(g, _bc(case), precision=sb.OF_MIXED if case.get("mixed") else sb.OF_FP64)
    if kind in ("advect", "adi", "project"):
        s["vel"] = [_host(inp[k]) for k in "uvw"]
        if kind == "advect":
            s["out"] = [g.zeros(k) for k in "uvw"]
        return s
    s["params"] = _params(case)
    state = {k: _host(inp[k], pinned=True) for k in "uvwp"}
    state.update({"adv_" + k: _host_zeros(g, k) for k in "uvw"})
    s["state"] = state
    if kind == "steps":
        s["saved"] = {k: _host_zeros(g, loc) for k, loc in
                      zip(("u", "v", "w", "adv_u", "adv_v", "adv_w", "p"), "uvwuvwp")}
    if kind == "adjoint":
        s["target"] = [_host(inp[k]) for k in ("tu", "tv", "tw")]
    return s


def _upload(s):
    st = s["state"]
    s["ctx"].upload_state(st["u"], st["v"], st["w"], st["adv_u"], st["adv_v"], st["adv_w"], st["p"])


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "rhs":
        norms = s["norms"] if case["norms"] else None
        _capi.check(s["lib"].of_pressure_rhs_noalloc(
            ctypes.byref(s["of_grid"]), s["dt"], 1.0, s["u"].data_ptr(), s["v"].data_ptr(), s["w"].data_ptr(),
            s["rhs"].data_ptr(), norms, torch.cuda.current_stream().cuda_stream))
        return [s["rhs"], norms[0], norms[1]] if case["norms"] else [s["rhs"]]
    if kind == "advect":
        return s["ctx"].compute_advection_term(*s["vel"], out=s["out"])
    if kind == "adi":
        out, lines = s["ctx"].solve_predictor_adi(s["vel"], _alpha(case))
        return list(out) + [lines]
    if kind == "poisson":
        p, diag = s["ctx"].solve_pressure_poisson(s["rhs"], s["pbc"], 400, case["tol"])
        return [p, diag["initial_residual_l2"]]
    if kind == "project":
        vel, phi, rhs, diag = s["ctx"].project_velocity(s["vel"], _dt(case), 1.0, 400, case["tol"])
        return list(vel) + [phi, rhs, diag["divergence_l2_before"], diag["rhs_l2"]]
    if kind == "steps":
        # from one saved state to the next
        _upload(s)
        s["ctx"].run_steps(s["params"], case["steps"])
        m = s["ctx"].download_state_into(s["saved"])
        return [s["saved"][k] for k in ("u", "v", "w", "adv_u", "adv_v", "adv_w", "p")] + [m["max_cfl"]]
    if kind == "step_host":
        m = s["ctx"].step_host(s["params"], s["state"])
        return [s["state"][k] for k in ("u", "v", "w", "adv_u", "adv_v", "adv_w", "p")] + [m["max_cfl"]]
    _upload(s)
    grad, info = s["ctx"].adjoint_gradient(s["params"], case["steps"], s["target"], checkpoint_every=case["every"])
    return list(grad) + [info["loss"], info["grad_viscosity"]]


def _alpha(case):
    return 0.5 * 0.01 * _dt(case) * 8.0  # a viscous predictor: alpha / h^2 of some hundredths


# Pressure iterations a solve takes on these flows, for the work a path cannot
# do without; one iteration of multigrid-preconditioned CG reads and writes the
# vectors of the fine level about 12 times when nothing is passed over twice.
_ITERATIONS = {1e-8: 10, 1e-10: 14, 1e-12: 20}


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    it = _ITERATIONS.get(case.get("tol"), 0)
    solve_b, solve_f = 8 * 12 * n * it, 120 * n * it
    kind = case["kind"]
    if kind == "rhs":
        return {"bytes": 8 * 4 * n, "flops": 10 * n}
    if kind in ("advect", "adi"):
        return {"bytes": 8 * 6 * n, "flops": (150 if kind == "advect" else 70) * n}
    if kind == "poisson":
        return {"bytes": 8 * 2 * n + solve_b, "flops": solve_f}
    if kind == "project":
        return {"bytes": 8 * 8 * n + solve_b, "flops": 30 * n + solve_f}
    if case.get("mixed"):
        solve_b //= 2
    step_b, step_f = 8 * 24 * n + solve_b, 400 * n + solve_f
    if kind == "adjoint":  # the forward pass, its recomputation and the reverse steps
        return {"bytes": 3 * case["steps"] * step_b, "flops": 3 * case["steps"] * step_f}
    return {"bytes": 8 * 14 * n + case.get("steps", 1) * step_b, "flops": case.get("steps", 1) * step_f}


# ---------------------------------------------------------------------------
# exact: plain FP64 torch
# ---------------------------------------------------------------------------
# Fields are padded tensors indexed [z, y, x]; axis a of (x, y, z) is dim 2 - a.

def _act(t):
    return t[1:-1, 1:-1, 1:-1]


def _component_bc(case, f, comp):
    types = FLOWS[case["flow"]]
    for a in range(3):
        others = [slice(1, -1)] * 3
        others[2 - a] = slice(None)
        t = f[tuple(others)].transpose(0, 2 - a) if a != 2 else f[tuple(others)]
        n = t.shape[0] - 2
        if types[2 * a] == PER:
            if comp == a:
                shared = 0.5 * (t[1] + t[n])
                t[1] = shared
                t[n] = shared
                t[0] = t[n - 1]
                t[n + 1] = t[2]
            else:
                t[0] = t[n]
                t[n + 1] = t[1]
            continue
        for side in range(2):
            ty = types[2 * a + side]
            b, gh, inner = (1, 0, 2) if side == 0 else (n, n + 1, n - 1)
            value = LID_VELOCITY[comp] if ty == LID else 0.0
            if comp == a:
                t[b] = value
                t[gh] = 2.0 * value - t[inner]
            elif ty in (WALL, LID):
                t[gh] = 2.0 * value - t[b]
            else:
                t[gh] = t[b]


def _tvd(vel, left, right, far_left, far_right):
    up = vel >= 0
    delta = right - left
    num = torch.where(up, left - far_left, far_right - right)
    tiny = delta.abs() < 1e-14
    r = torch.where(tiny, torch.zeros_like(delta), num / torch.where(tiny, torch.ones_like(delta), delta))
    half = 0.5 * (r + r.abs()) / (1.0 + r.abs()) * delta
    muscl = torch.where(up, left + half, right - half)
    far_ok = torch.where(up, torch.isfinite(far_left), torch.isfinite(far_right))
    return torch.where((vel.abs() < 1e-14) | ~far_ok, torch.where(up, left, right), muscl)


def _advection(g, vel):
    h = (g.dx, g.dy, g.dz)
    out = []
    for c in range(3):
        f = vel[c]
        # two more layers whose values mark "outside the storage"
        e = torch.full([n + 2 for n in f.shape], math.nan, dtype=f.dtype, device=f.device)
        e[1:-1, 1:-1, 1:-1] = f
        total = 0.0
        for d in range(3):
            win = {}
            for k in range(-2, 3):
                t = e
                for a in range(3):
                    o = k if a == d else 0
                    t = t.narrow(2 - a, 2 + o, f.shape[2 - a] - 2)
                win[k] = t
            if d == c:
                lo_v = 0.5 * (win[-1] + win[0])
                hi_v = 0.5 * (win[0] + win[1])
            else:
                # the other component's faces, at this component's points
                fd, n = vel[d], [f.shape[2 - a] - 2 for a in range(3)]

                def at(oc, od):
                    t = fd
                    for a in range(3):
                        o = oc if a == c else od if a == d else 0
                        t = t.narrow(2 - a, 1 + o, n[a])
                    return t

                lo_v = 0.5 * (at(-1, 0) + at(0, 0))
                hi_v = 0.5 * (at(-1, 1) + at(0, 1))
            lo = _tvd(lo_v, win[-1], win[0], win[-2], win[1])
            hi = _tvd(hi_v, win[0], win[1], win[-1], win[2])
            total = total + (hi_v * hi - lo_v * lo) / h[d]
        r = torch.zeros_like(f)
        _act(r)[...] = total
        out.append(r)
    return out


def _line_matrix(case, g, comp, a, alpha):
    """(matrix, rhs constants, first, one past the last storage index, duplicate) of one line solve."""
    types = FLOWS[case["flow"]]
    n_act = (g.nx, g.ny, g.nz)[a] + (1 if comp == a else 0)
    beta = alpha / (g.dx, g.dy, g.dz)[a] ** 2
    begin, end = 1, 1 + n_act
    per = types[2 * a] == PER
    if per and comp == a:
        end -= 1
    elif comp == a:
        begin, end = begin + 1, end - 1
    n = end - begin
    if n <= 0:
        return None
    m = torch.zeros((n, n), dtype=torch.float64, device=_device())
    i = torch.arange(n, device=m.device)
    m[i, i] = 1.0 + 2.0 * beta
    if n > 1:
        m[i[1:], i[:-1]] -= beta
        m[i[:-1], i[1:]] -= beta
    add = [0.0, 0.0]
    if per:
        if n == 1:
            m[0, 0] -= 2.0 * beta
        else:
            m[0, n - 1] -= beta
            m[n - 1, 0] -= beta
    else:
        for side, q in ((0, 0), (1, n - 1)):
            ty = types[2 * a + side]
            value = LID_VELOCITY[comp] if ty == LID else 0.0
            if comp == a:
                add[side] += beta * value
            elif ty in (WALL, LID):
                m[q, q] += beta
                add[side] += beta * 2.0 * value
            else:
                m[q, q] -= beta
    return m, add, begin, end, per and comp == a


def _adi(case, g, rhs, alpha):
    out = []
    for c in range(3):
        f = rhs[c].clone()
        _component_bc(case, f, c)
        for a in range(3):
            lm = _line_matrix(case, g, c, a, alpha)
            if lm is not None:
                m, add, begin, end, dup = lm
                act = f[tuple(slice(None) if 2 - a == d else slice(1, -1) for d in range(3))]
                t = act.movedim(2 - a, 0)
                r = t[begin:end].reshape(end - begin, -1).clone()
                r[0] += add[0]
                r[-1] += add[1]
                x = torch.linalg.solve(m, r).reshape(t[begin:end].shape)
                t[begin:end] = x
                if dup:
                    t[end] = x[0]
            _component_bc(case, f, c)
        out.append(f)
    return out


def _laplacian_1d(n, h, lo, hi):
    """-d2/dx2 on n cells with homogeneous boundary rules."""
    m = torch.zeros((n, n), dtype=torch.float64, device=_device())
    for i in range(n):
        m[i, i] += 2.0
        for j, ty in ((i - 1, lo), (i + 1, hi)):
            if 0 <= j < n:
                m[i, j] -= 1.0
            elif ty == sb.P_PERIODIC:
                m[i, j % n] -= 1.0
            else:
                m[i, i] += 1.0 if ty == sb.P_DIRICHLET else -1.0
    return m / (h * h)


def _poisson(g, pbc, rhs):
    """Solves Lap x = rhs on the cells (zero mean where the problem is singular)."""
    lam, q = [], []
    for a, (n, h) in enumerate(((g.nx, g.dx), (g.ny, g.dy), (g.nz, g.dz))):
        m = _laplacian_1d(n, h, pbc[2 * a], pbc[2 * a + 1]).cpu()
        e, v = torch.linalg.eigh(m)
        lam.append(e.to(rhs.device))
        q.append(v.to(rhs.device))
    b = -rhs
    singular = sb.P_DIRICHLET not in pbc
    if singular:
        b = b - b.mean()
    t = torch.einsum("zyx,xi->zyi", b, q[0])
    t = torch.einsum("zyi,yj->zji", t, q[1])
    t = torch.einsum("zji,zk->kji", t, q[2])
    den = lam[0].reshape(1, 1, -1) + lam[1].reshape(1, -1, 1) + lam[2].reshape(-1, 1, 1)
    if singular:
        t.view(-1)[den.reshape(-1).abs().argmin()] = 0.0
        den = torch.where(den.abs() == den.abs().min(), torch.ones_like(den), den)
    t = t / den
    t = torch.einsum("kji,zk->zji", t, q[2])
    t = torch.einsum("zji,yj->zyi", t, q[1])
    t = torch.einsum("zyi,xi->zyx", t, q[0])
    return t - t.mean() if singular else t


def _divergence(g, v):
    return ((v[0][1:-1, 1:-1, 2:-1] - v[0][1:-1, 1:-1, 1:-2]) / g.dx +
            (v[1][1:-1, 2:-1, 1:-1] - v[1][1:-1, 1:-2, 1:-1]) / g.dy +
            (v[2][2:-1, 1:-1, 1:-1] - v[2][1:-2, 1:-1, 1:-1]) / g.dz)


def _pressure_types(case):
    return tuple(sb.P_PERIODIC if t == PER else sb.P_NEUMANN for t in FLOWS[case["flow"]])


def _correct(case, g, pred, phi, scale):
    """pred + scale grad(phi) on the active faces, ghosts filled."""
    types = _pressure_types(case)
    out = []
    for a, h in enumerate((g.dx, g.dy, g.dz)):
        d = 2 - a
        first, last = phi.narrow(d, 0, 1), phi.narrow(d, phi.shape[d] - 1, 1)
        lo, hi = (last, first) if types[2 * a] == sb.P_PERIODIC else (first, last)
        e = torch.cat((lo, phi, hi), d)
        n = e.shape[d] - 1
        f = pred[a].clone()
        _act(f)[...] += scale * (e.narrow(d, 1, n) - e.narrow(d, 0, n)) / h
        _component_bc(case, f, a)
        out.append(f)
    return out


def _second(t, a, h, n):
    """Second difference along axis a over the active window of the other axes."""
    d = 2 - a
    return (t.narrow(d, 2, n) - 2.0 * t.narrow(d, 1, n) + t.narrow(d, 0, n)) / (h * h)


def _mixed_second(f, axes, h):
    t = f
    for a in range(3):
        d = 2 - a
        n = t.shape[d] - 2
        t = _second(t, a, h[a], n) if a in axes else t.narrow(d, 1, n)
    return t


def _total_pressure_bc(case, g, vel, nu, p):
    types, h = FLOWS[case["flow"]], (g.dx, g.dy, g.dz)
    for a in range(3):
        others = [slice(1, -1)] * 3
        others[2 - a] = slice(None)
        t = p[tuple(others)].movedim(2 - a, 0)
        n = t.shape[0] - 2
        if types[2 * a] == PER:
            t[0] = t[n]
            t[n + 1] = t[1]
            continue
        dif = nu * sum(_mixed_second(vel[a], (b,), h) for b in range(3))
        dif = dif.movedim(2 - a, 0)
        t[0] = t[1] - dif[0] * h[a]
        t[n + 1] = t[n] + dif[-1] * h[a]


def _step(case, g, st):
    """One projection step of {vel, adv (or None), p}; returns the next state and the CFL number."""
    dt, nu, h = _dt(case), case["nu"], (g.dx, g.dy, g.dz)
    alpha = 0.5 * nu * dt
    cur = [f.clone() for f in st["vel"]]
    for c in range(3):
        _component_bc(case, cur[c], c)
    adv = _advection(g, cur)
    rhs = []
    for c in range(3):
        f = cur[c]
        lap = sum(_mixed_second(f, (b,), h) for b in range(3))
        d = 2 - c
        pe = st["p"][tuple(slice(None) if x == d else slice(1, -1) for x in range(3))]
        n = pe.shape[d] - 1
        gp = (pe.narrow(d, 1, n) - pe.narrow(d, 0, n)) / h[c]
        corr = _mixed_second(f, (0, 1), h)
        if case["flow"] != "cavity" and g.nz != 1:
            corr = corr + _mixed_second(f, (0, 2), h) + _mixed_second(f, (1, 2), h) - \
                alpha * _mixed_second(f, (0, 1, 2), h)
        r = _act(f) - dt * gp + 0.5 * dt * nu * lap + alpha * alpha * corr
        if st["adv"] is None:
            r = r - dt * _act(adv[c])
        else:
            r = r - 1.5 * dt * _act(adv[c]) + 0.5 * dt * _act(st["adv"][c])
        full = st["vel"][c].clone()
        _act(full)[...] = r
        rhs.append(full)
    pred = _adi(case, g, rhs, alpha)
    q = _divergence(g, pred) / dt
    phi = _poisson(g, _pressure_types(case), q)
    vel = _correct(case, g, pred, phi, -dt)
    p = st["p"].clone()
    _act(p)[...] += phi - 0.5 * nu * dt * q
    _total_pressure_bc(case, g, vel, nu, p)
    cc = [0.5 * (_act(v).narrow(2 - a, 0, _act(v).shape[2 - a] - 1) + _act(v).narrow(2 - a, 1, _act(v).shape[2 - a] - 1))
          for a, v in enumerate(vel)]
    cfl = dt * sum(c.abs() / hh for c, hh in zip(cc, h)).max()
    return {"vel": vel, "adv": adv, "p": p}, float(cfl)


def exact(case, seed):
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "adjoint" or cells * case.get("steps", 1) > 8 * 2 ** 24:
        return None
    g = _grid(case)
    inp = _inputs(case, seed)
    if kind == "poisson":
        pbc = PRESSURE[case["flow"]]
        rhs = _act(inp["rhs"])
        b = rhs - rhs.mean() if sb.P_DIRICHLET not in pbc else rhs
        out = inp["pressure"].clone()
        _act(out)[...] = _poisson(g, pbc, rhs)
        return [out, float(b.square().mean().sqrt())]
    vel = [inp[k] for k in "uvw"]
    if kind == "rhs":
        div = _divergence(g, vel)
        out = torch.zeros_like(inp["p"])
        _act(out)[...] = div / _dt(case)
        if not case["norms"]:
            return [out]
        return [out, float(div.square().mean().sqrt()), float((div / _dt(case)).square().mean().sqrt())]
    if kind == "advect":
        return _advection(g, vel)
    if kind == "adi":
        return _adi(case, g, vel, _alpha(case)) + [None]
    if kind == "project":
        dt = _dt(case)
        for c in range(3):
            _component_bc(case, vel[c], c)
        div = _divergence(g, vel)
        phi = torch.zeros_like(inp["p"])
        _act(phi)[...] = _poisson(g, _pressure_types(case), div / dt)
        rhs = torch.zeros_like(inp["p"])
        _act(rhs)[...] = div / dt
        return _correct(case, g, vel, _act(phi), -dt) + [phi, rhs, float(div.square().mean().sqrt()),
                                                         float((div / dt).square().mean().sqrt())]
    st = {"vel": vel, "adv": None, "p": inp["p"]}
    cfl = 0.0
    for _ in range(case.get("steps", 1)):
        st, cfl = _step(case, g, st)
    return st["vel"] + st["adv"] + [st["p"], cfl]

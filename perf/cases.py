"""The work whose speed counts: what programs that use this package have it do.

A case is a plain dict.  ``kind`` says which public entry point it goes through:

``evolve``  ``ClawSolver2D.evolve_to_time`` on a problem whose state lives on the GPU (what
            ``Controller.run`` calls between two output times): ghost cells, step, Courant number,
            dt choice and accept/reject of every step.  A pass restarts from a copy of the initial
            planes that the program keeps on the GPU and ends with its copy of the result.
``batch``   ``batch.Batch``: an ensemble of independent problems uploaded, run and downloaded.
``train``   ``learned.Network.train``: forward, backward and Adam over a sample set.
``host``    ``classic2.step2`` / ``step2ds``: one step on host arrays, as the reference's own
            ``ClawSolver2D.step_hyperbolic`` calls its Fortran module.

``exact`` recomputes the outputs with plain torch in 64 bits: the wave-propagation algorithm
written on whole arrays (LeVeque, Finite Volume Methods for Hyperbolic Problems, 2002).
"""
import math
import random

import numpy as np
import torch

import pyclaw_b200 as pyclaw
from pyclaw_b200 import batch, classic2, learned, riemann, workloads
from pyclaw_b200.geometry import Dimension, Domain
from pyclaw_b200.slabs import DevicePlanes
from pyclaw_b200.solution import Solution
from pyclaw_b200.state import State

GAMMA, GRAV = 1.4, 1.0
RHO, BULK = 1.0, 4.0  # the homogeneous acoustic medium: c = 2, Z = 2
LIMITERS = {"minmod": 1, "superbee": 2, "vanleer": 3, "MC": 4}
BCS = {"extrap": pyclaw.BC.extrap, "periodic": pyclaw.BC.periodic, "wall": pyclaw.BC.wall}
# Riemann solver, components, waves, domain, and FP64 operations of one cell-update: what the solves of
# its two interfaces, the limiter, the corrections and (unsplit) the four transverse solves need
SOLVERS = {
    "advection": (riemann.advection_2D, 1, 1, (0.0, 1.0), 60),
    "acoustics": (riemann.acoustics_2D, 3, 2, (-1.0, 1.0), 250),
    "vc_acoustics": (riemann.vc_acoustics_2D, 3, 2, (-1.0, 1.0), 300),
    "shallow": (riemann.shallow_roe_with_efix_2D, 3, 3, (-2.5, 2.5), 600),
    "euler": (riemann.euler_4wave_2D, 4, 4, (0.0, 1.0), 1100),
    "euler_exact": (riemann.euler_exact_2D, 4, 3, (0.0, 1.0), 2000),
}


def _evolve(name, solver, mx, my, steps, split=False, trans=2, limiter="MC", bc="extrap", cfl=0.9, learned=False):
    return {"name": name, "kind": "evolve", "solver": solver, "mx": mx, "my": my, "steps": steps, "split": split,
            "trans": trans, "limiter": limiter, "bc": bc, "cfl": cfl, "learned": learned}


def listed():
    return [
        # the homogeneous acoustics example, whole: 100^2, split, CFL 0.45, 27 steps.  The smallest runs
        # (examples, teaching, parameter scans): launches and latency
        _evolve("acoustics 100 split", "acoustics", 100, 100, 27, split=True, cfl=0.45),
        # the walled acoustics benchmark, whole: 200^2, unsplit, to t = 0.6 in 134 steps
        _evolve("acoustics 200 wall", "acoustics", 200, 200, 134, bc="wall"),
        # a ragged Euler quadrant problem with the solver's defaults: dimensional splitting, minmod
        _evolve("euler 353x271 split", "euler", 353, 271, 40, split=True, limiter="minmod"),
        # the headline: the Euler quadrant benchmark at 1024^2, a stretch of its run
        _evolve("euler 1024", "euler", 1024, 1024, 24),
        # unsplit with the default transverse mode and another limiter, a wide odd grid
        _evolve("euler 1291x433 inc", "euler", 1291, 433, 16, trans=1, limiter="superbee"),
        # the largest: the shallow-water dam break at 4096^2
        _evolve("shallow 4096", "shallow", 4096, 4096, 6),
        # two materials, aux data on the device, the default transverse mode, walls (acoustics_variable)
        _evolve("vc acoustics 400", "vc_acoustics", 400, 400, 40, trans=1, bc="wall"),
        # the exact Riemann solver, Newton from its own guess
        _evolve("exact 1024", "euler_exact", 1024, 1024, 6),
        # the exact solver's benchmark size, Newton from the trained network's guess
        _evolve("exact 2048 learned", "euler_exact", 2048, 2048, 3, learned=True),
        # an ensemble of uneven quadrant problems from host arrays, its 100 steps, and read back
        {"name": "batch 24", "kind": "batch", "n": 24, "lo": 64, "hi": 512, "steps": 100},
        # one epoch over 2^20 samples in minibatches of 16384 (the network's training set is 2^24, 16 epochs)
        {"name": "train 2^20", "kind": "train", "samples": 1 << 20, "batch": 16384, "epochs": 1},
        # one unsplit step through the drop-in for the reference's Fortran module
        {"name": "host step2 500", "kind": "host", "solver": "euler", "mx": 500, "my": 500, "split": False, "trans": 2,
         "limiter": "MC", "bc": "extrap", "cfl": 0.9},
    ]


MOST = 4096 * 4096 * 6 * 600  # FP64 operations of the largest listed case


def draw(rng):
    kind = rng.choice(["evolve"] * 6 + ["batch", "train", "host"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "batch":
        lo = rng.randrange(48, 128)
        return {"kind": kind, "n": rng.randrange(6, 25), "lo": lo, "hi": rng.randrange(lo + 16, 481),
                "steps": rng.randrange(30, 101)}
    if kind == "train":
        b = size(2000, 32000)
        return {"kind": kind, "samples": b * rng.randrange(6, 40) + rng.randrange(b), "batch": b, "epochs": 1}
    solver = rng.choice(["advection", "acoustics", "vc_acoustics", "shallow", "shallow", "euler", "euler", "euler"])
    c = {"kind": kind, "solver": solver, "split": rng.random() < 0.4, "trans": rng.choice([1, 2, 2]),
         "limiter": rng.choice(sorted(LIMITERS)), "bc": rng.choice(sorted(BCS)), "cfl": 0.9}
    if kind == "host":
        c |= {"solver": rng.choice(["acoustics", "shallow", "euler"]), "bc": "extrap"}
        if c["limiter"] == "vanleer":
            c["limiter"] = "minmod"
        return {**c, "mx": size(40, 700), "my": size(40, 700)}
    c["learned"] = False
    if solver in ("euler", "shallow") and c["limiter"] == "vanleer":
        c["limiter"] = "MC"  # (van Leer's is the linear examples' limiter)
    if c["solver"] == "euler":
        c["bc"] = "extrap"  # (the quadrant states part too fast at a wall or across a periodic edge)
    if rng.random() < 0.2:
        c |= {"solver": "euler_exact", "split": False, "trans": 2, "bc": "extrap", "learned": rng.random() < 0.5,
              "limiter": rng.choice(["MC", "minmod", "superbee"])}
    c["mx"], c["my"] = size(50, 2600), size(50, 2600)
    room = MOST / (c["mx"] * c["my"] * SOLVERS[c["solver"]][4])
    c["steps"] = max(1, min(rng.randrange(4, 61), int(0.8 * room)))
    return c


# ---- inputs ---------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _centers(n, lo, hi):
    return lo + (torch.arange(n, dtype=torch.float64, device=_device()) + 0.5) * ((hi - lo) / n)


def _waves(r, x, y, amp, x0, y0, radius):
    """A smooth field of a few random modes that is exactly zero outside a disc."""
    s = ((x - x0) ** 2 + (y - y0) ** 2) / radius ** 2
    bump = (1.0 - s).clamp_min(0.0) ** 3
    f = torch.zeros_like(s)
    for _ in range(5):
        kx, ky, ph = r.uniform(-6, 6) / radius, r.uniform(-6, 6) / radius, r.uniform(0, 6.28)
        f += torch.sin(kx * x + ky * y + ph)
    return amp * bump * f / 3.0


def _euler_q(rho, u, v, p):
    return torch.stack([rho, rho * u, rho * v, 0.5 * rho * (u * u + v * v) + p / (GAMMA - 1.0)])


def _initial(case, seed):
    """q as [component, row, column] on the GPU, and aux (or None)."""
    r = random.Random(int(seed))
    name = case["solver"]
    lo, hi = SOLVERS[name][3]
    x, y = _centers(case["mx"], lo, hi)[None, :], _centers(case["my"], lo, hi)[:, None]
    if name == "advection":  # the square of the advection example, moved and scaled
        a, b = r.uniform(0.05, 0.2), r.uniform(0.05, 0.2)
        q = r.uniform(0.7, 1.1) * ((x > a) & (x < a + 0.5) & (y > b) & (y < b + 0.5)).double() + 0.1
        return q[None] + _waves(r, x, y, 0.1, 0.5, 0.5, 0.3)[None], None
    if name == "acoustics":  # the pulse of the walled benchmark
        p = torch.exp(-100.0 * ((x - r.uniform(0.1, 0.4)) ** 2 + (y - r.uniform(-0.2, 0.2)) ** 2))
        return torch.stack([p, torch.zeros_like(p), torch.zeros_like(p)]), None
    if name == "vc_acoustics":  # a pressure ring beside a material interface
        d = torch.sqrt((x - r.uniform(-0.6, -0.4)) ** 2 + (y - r.uniform(-0.1, 0.1)) ** 2)
        p = (torch.abs(d - 0.25) <= 0.1).double() * (1.0 + torch.cos(math.pi * (d - 0.25) / 0.1))
        left = (x < 0.0).double() + 0.0 * y
        aux = torch.stack([4.0 * left + 1.0 * (1.0 - left), 1.0 * left + 2.0 * (1.0 - left)])
        return torch.stack([p, torch.zeros_like(p), torch.zeros_like(p)]), aux
    if name == "shallow":  # the dam break some time after the break: a disturbed disc, the rest at rest
        x0, y0 = r.uniform(-0.1, 0.1), r.uniform(-0.1, 0.1)
        d = torch.sqrt((x - x0) ** 2 + (y - y0) ** 2)
        h = 1.0 + (d < r.uniform(0.45, 0.55)).double() + _waves(r, x, y, 0.15, x0, y0, 1.2)
        hu, hv = _waves(r, x, y, 0.3, x0, y0, 1.2), _waves(r, x, y, 0.3, x0, y0, 1.2)
        return torch.stack([h, hu, hv]), None
    # Euler: the quadrant problem in the middle of its run: the four states, wavy fronts between them, a
    # disturbed disc around the corner point and constant states outside it
    xs, ys = r.uniform(0.66, 0.74), r.uniform(0.66, 0.74)
    fx = xs + 0.05 * torch.sin(9.0 * y + r.uniform(0, 6)) * torch.exp(-(((y - ys) / 0.3) ** 2))
    fy = ys + 0.05 * torch.sin(9.0 * x + r.uniform(0, 6)) * torch.exp(-(((x - xs) / 0.3) ** 2))
    east, north = (x >= fx), (y >= fy)
    rho, u, v, p = (torch.zeros_like(x + y) for _ in range(4))
    for k, m in (("NE", east & north), ("NW", ~east & north), ("SW", ~east & ~north), ("SE", east & ~north)):
        f = r.uniform(0.97, 1.03)
        for z, val in zip((rho, u, v, p), workloads.QUADRANT_STATES[k]):
            z += m.double() * (val * f)
    rho = rho * (1.0 + _waves(r, x, y, 0.2, 0.55, 0.55, 0.45))
    p = p * (1.0 + _waves(r, x, y, 0.2, 0.55, 0.55, 0.45))
    u, v = u + _waves(r, x, y, 0.2, 0.55, 0.55, 0.45), v + _waves(r, x, y, 0.2, 0.55, 0.55, 0.45)
    return _euler_q(rho, u, v, p), None


def _host(a):
    """[component, row, column] on the GPU -> the package's (component, x, y) in Fortran order."""
    return a.permute(1, 2, 0).contiguous().cpu().numpy().T


def _spacing(case):
    lo, hi = SOLVERS[case["solver"]][3]
    return (hi - lo) / case["mx"], (hi - lo) / case["my"]


def _first_dt(case, q):
    """dt of Courant number `cfl` for the cells' own speeds."""
    name, (dx, dy) = case["solver"], _spacing(case)
    if name == "advection":
        sx, sy = 0.5, 1.0
    elif name in ("acoustics", "vc_acoustics"):
        sx = sy = 2.0
    else:
        c = torch.sqrt(GRAV * q[0]) if name == "shallow" else torch.sqrt(
            GAMMA * (GAMMA - 1.0) * (q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) / q[0]) / q[0])
        sx, sy = float((torch.abs(q[1] / q[0]) + c).max()), float((torch.abs(q[2] / q[0]) + c).max())
    return case["cfl"] / max(sx / dx, sy / dy)


def _problem_data(name):
    if name == "advection":
        return {"u": 0.5, "v": 1.0}
    if name == "acoustics":
        return {"rho": RHO, "bulk": BULK, "cc": math.sqrt(BULK / RHO), "zz": RHO * math.sqrt(BULK / RHO)}
    return {} if name == "vc_acoustics" else {"grav": GRAV} if name == "shallow" else {"gamma": GAMMA}


def _network(seed, samples, batch_size, epochs):
    net = learned.Network(seed=seed)
    net.generate(samples, seed=seed)
    if epochs:
        net.train(epochs, batch_size, 3e-3)
    return net


def _prepare_evolve(case, seed):
    rp, meqn, mwaves, (lo, hi), _ = SOLVERS[case["solver"]]
    q, aux = _initial(case, seed)
    solver = pyclaw.ClawSolver2D(rp)
    solver.num_waves = mwaves
    solver.dimensional_split = case["split"]
    solver.transverse_waves = case["trans"]
    solver.limiters = LIMITERS[case["limiter"]]
    solver.cfl_desired, solver.cfl_max = case["cfl"], (1.0 if case["cfl"] > 0.5 else 0.5)
    solver.all_bcs = BCS[case["bc"]]
    domain = Domain([Dimension(lo, hi, case["mx"], name="x"), Dimension(lo, hi, case["my"], name="y")])
    state = State(domain, meqn, 0 if aux is None else aux.shape[0])
    state.problem_data.update(_problem_data(case["solver"]))
    state.q = _host(q)
    if aux is not None:
        state.aux[...] = _host(aux)
        solver.aux_bc_lower = [BCS[case["bc"]]] * 2
        solver.aux_bc_upper = [BCS[case["bc"]]] * 2
    solution = Solution(state, domain)
    solver.setup(solution)
    stream = torch.cuda.Stream()  # the solver's work and the program's copies share it
    solver._dev.set_stream(stream.cuda_stream)
    if case["learned"]:
        learned.attach(solver, _network(seed, 1 << 20, 16384, 2))
    dt = _first_dt(case, q)
    torch.cuda.synchronize()
    return {"kind": "evolve", "solver": solver, "solution": solution, "stream": stream, "dt": dt, "cfl": case["cfl"],
            "tend": (case["steps"] - 0.5) * dt, "start": DevicePlanes(solver._dev).t.clone(),
            "mx": case["mx"], "my": case["my"]}


def _run_evolve(s):
    solver, solution = s["solver"], s["solution"]
    with torch.cuda.stream(s["stream"]):
        DevicePlanes(solver._dev).t.copy_(s["start"])
    solution.t = 0.0
    solver.dt, solver.dt_old = s["dt"], None
    solver.status["numsteps"] = 0
    status = solver.evolve_to_time(solution, s["tend"])
    with torch.cuda.stream(s["stream"]):  # the program's own copy of the result: it outlives the solver
        q = DevicePlanes(solver._dev).t[:, 2:s["my"] + 2, 2:s["mx"] + 2].clone()
    return {"q": q, "t": solution.t, "dt": solver.dt, "cfl": solver.cfl.get_cached_max(), "steps": status["numsteps"]}


def _sides(case):
    n = case["n"]
    return [int(round(case["lo"] + (case["hi"] - case["lo"]) * ((k * 53) % n) / (n - 1))) for k in range(n)]


def _ensemble(case, seed):
    """The batched workload's quadrant data: per problem (side, split point, four states, first dt)."""
    r, out = np.random.default_rng(int(seed)), []
    for side in _sides(case):
        split = tuple(r.uniform(0.3, 0.7, 2))
        st = {k: (*r.uniform(0.5, 2.0, 1), *r.uniform(-0.5, 0.5, 2), *r.uniform(0.5, 2.0, 1))
              for k in ("NE", "NW", "SW", "SE")}
        smax = max(max(abs(u), abs(v)) + math.sqrt(GAMMA * p / rho) for rho, u, v, p in st.values())
        out.append((side, split, st, 0.45 / side / smax))
    return out


def _prepare_batch(case, seed):
    claws = []
    for side, split, st, dt in _ensemble(case, seed):
        claw = workloads.euler_quadrants_unsplit(n=side, split=split, states=st)
        claw.solver.dt_initial = dt
        claws.append(claw)
    return {"kind": "batch", "batch": batch.Batch(claws), "dt": [c.solver.dt_initial for c in claws],
            "steps": case["steps"]}


def _run_batch(s):
    b = s["batch"]
    b.upload()
    b.set_time(s["dt"], 0.0, 1e99, 0.9, 1.0, 1e99)
    b.run(s["steps"])
    st = b.state()
    return {"q": [b.q(i) for i in range(b.n)], "t": st["t"], "dt": st["dt"], "nsteps": st["nsteps"],
            "nreject": st["nreject"]}


def _weights(seed):
    r = np.random.default_rng(int(seed) + 1)
    p = np.zeros(learned.NPARAM)
    for off, n, fan in ((0, 192, 38), (224, 1024, 64), (1280, 32, 33)):  # W1, W2, W3; zero biases
        p[off:off + n] = r.uniform(-1.0, 1.0, n) * math.sqrt(6.0 / fan)
    return p.astype(np.float32)


def _prepare_train(case, seed):
    net = _network(seed, case["samples"], case["batch"], 0)
    net.params = _weights(seed)
    return {"kind": "train", "net": net, "epochs": case["epochs"], "batch": case["batch"]}


def _run_train(s):
    loss = s["net"].train(s["epochs"], s["batch"], 3e-3)
    return {"params": s["net"].params, "loss": loss}


def _prepare_host(case, seed):
    q, _ = _initial(case, seed)
    for k, v in _problem_data(case["solver"]).items():
        setattr(classic2.cparam, k, v)
    rp, meqn, mwaves, _, _ = SOLVERS[case["solver"]]
    qbc = _host(_fill(q, case["bc"], 1.0))
    method = np.array([1, 2, -1 if case["split"] else case["trans"], 0, 0, 0, 0])
    return {"kind": "host", "case": case, "qbc": qbc, "rp": rp, "dt": _first_dt(case, q), "method": method,
            "mthlim": np.full(mwaves, LIMITERS[case["limiter"]])}


def _run_host(s):
    c, rp = s["case"], s["rp"]
    mx, my, (dx, dy) = c["mx"], c["my"], _spacing(s["case"])
    qold = s["qbc"].copy(order="F")
    lead = (max(mx, my), 2, mx, my)
    tail = (None, dx, dy, s["dt"], s["method"], s["mthlim"], None, None, None, None)
    if c["split"]:
        q, cx = classic2.step2ds(*lead, qold, s["qbc"], *tail, 1, False, rp, rp)
        q, cy = classic2.step2ds(*lead, q, q, *tail, 2, False, rp, rp)
        cfl = max(cx, cy)
    else:
        q, cfl = classic2.step2(*lead, qold, s["qbc"], *tail, False, rp, rp)
    return {"q": q[:, 2:-2, 2:-2], "cfl": cfl}


def prepare(case, seed):
    return {"evolve": _prepare_evolve, "batch": _prepare_batch, "train": _prepare_train,
            "host": _prepare_host}[case["kind"]](case, seed)


def run(state):
    return {"evolve": _run_evolve, "batch": _run_batch, "train": _run_train, "host": _run_host}[state["kind"]](state)


def work(case):
    if case["kind"] == "train":  # every sample's 8 floats and target; forward and backward of the two layers
        n = case["samples"] // case["batch"] * case["batch"] * case["epochs"]
        return {"bytes": n * 40.0, "flops": n * 7500.0}
    if case["kind"] == "batch":
        cells, (meqn, ops), steps = sum(s * s for s in _sides(case)), (4, SOLVERS["euler"][4]), case["steps"]
    else:
        cells, steps = case["mx"] * case["my"], case.get("steps", 1)
        meqn, ops = SOLVERS[case["solver"]][1], SOLVERS[case["solver"]][4] * (0.6 if case["split"] else 1.0)
    # q read and written once a step
    return {"bytes": 16.0 * meqn * cells * steps, "flops": float(ops) * cells * steps}


# ---- the same results from plain torch in 64 bits ----------------------------------------------
def _fill(q, bc, sign=-1.0):
    """[component, row, column] with two ghost cells on each side: columns first, then rows.  A wall
    mirrors, with the normal component negated when sign is -1."""
    for dim in (2, 1):
        n = q.shape[dim]
        if bc == "periodic":
            left, right = q.narrow(dim, n - 2, 2), q.narrow(dim, 0, 2)
        elif bc == "extrap":
            left = q.narrow(dim, 0, 1).repeat_interleave(2, dim)
            right = q.narrow(dim, n - 1, 1).repeat_interleave(2, dim)
        else:
            left, right = q.narrow(dim, 0, 2).flip(dim), q.narrow(dim, n - 2, 2).flip(dim)
            if sign < 0 and q.shape[0] > 2:
                left, right = left.clone(), right.clone()
                left[3 - dim] *= -1.0
                right[3 - dim] *= -1.0
        q = torch.cat([left, q, right], dim)
    return q


def _vec(m, parts):
    """A [component, ...] tensor from {component: value}, zero elsewhere."""
    like = next(iter(parts.values()))
    return torch.stack([parts[k] if k in parts else torch.zeros_like(like) for k in range(m)])


def _roe_split(s, w, s0, s1, s2, s3, efix):
    """Fluctuations of Roe's linearisation: waves by the sign of their speeds, the acoustic ones split where
    they are transonic rarefactions (Harten & Hyman).  s0/s1: the first characteristic speed left and right of
    the first wave; s2/s3: the last one left and right of the last wave."""
    if efix:
        first = torch.where((s0 < 0) & (s1 > 0), s0 * (s1 - s[0]) / (s1 - s0), s[0].clamp_max(0.0))
        last = torch.where((s2 < 0) & (s3 > 0), s2 * (s3 - s[-1]) / (s3 - s2), s[-1].clamp_max(0.0))
    am = first * w[0] + last * w[-1] + sum(x.clamp_max(0.0) * y for x, y in zip(s[1:-1], w[1:-1]))
    return am, sum(x * y for x, y in zip(s, w)) - am


def _rpn2(name, L, R, mu, auxL, auxR):
    """Waves, speeds, fluctuations, and what the transverse solver needs."""
    mv = 3 - mu
    d = R - L
    if name == "advection":
        s = torch.full_like(d[0], 0.5 if mu == 1 else 1.0)
        return [d], [s], s.clamp_max(0) * d, s.clamp_min(0) * d, None
    if name in ("acoustics", "vc_acoustics"):
        if name == "acoustics":
            c = math.sqrt(BULK / RHO)
            zl = zr = torch.full_like(d[0], RHO * c)
            cl = cr = torch.full_like(d[0], c)
        else:
            zl, zr, cl, cr = auxL[0] * auxL[1], auxR[0] * auxR[1], auxL[1], auxR[1]
        a1, a2 = (-d[0] + zr * d[mu]) / (zl + zr), (d[0] + zl * d[mu]) / (zl + zr)
        w = [_vec(3, {0: -a1 * zl, mu: a1}), _vec(3, {0: a2 * zr, mu: a2})]
        return w, [-cl, cr], -cl * w[0], cr * w[1], None
    if name == "shallow":
        rl, rr = torch.sqrt(L[0]), torch.sqrt(R[0])
        u = (L[mu] / rl + R[mu] / rr) / (rl + rr)
        v = (L[mv] / rl + R[mv] / rr) / (rl + rr)
        a = torch.sqrt(GRAV * 0.5 * (L[0] + R[0]))
        a1, a2, a3 = ((u + a) * d[0] - d[mu]) / (2 * a), d[mv] - v * d[0], (d[mu] - (u - a) * d[0]) / (2 * a)
        w = [_vec(3, {0: a1, mu: a1 * (u - a), mv: a1 * v}), _vec(3, {mv: a2}),
             _vec(3, {0: a3, mu: a3 * (u + a), mv: a3 * v})]
        s = [u - a, u, u + a]
        m1, m3 = L + w[0], R - w[2]
        am, ap = _roe_split(s, w, L[mu] / L[0] - torch.sqrt(GRAV * L[0]), m1[mu] / m1[0] - torch.sqrt(GRAV * m1[0]),
                            m3[mu] / m3[0] + torch.sqrt(GRAV * m3[0]), R[mu] / R[0] + torch.sqrt(GRAV * R[0]), True)
        return w, s, am, ap, (u, v, a)

    def prim(q):
        return q[0], q[mu] / q[0], q[mv] / q[0], (GAMMA - 1) * (q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) / q[0])

    (r_l, ul, vl, pl), (r_r, ur, vr, pr) = prim(L), prim(R)
    rl, rr = torch.sqrt(r_l), torch.sqrt(r_r)
    u, v = (rl * ul + rr * ur) / (rl + rr), (rl * vl + rr * vr) / (rl + rr)
    H = ((L[3] + pl) / rl + (R[3] + pr) / rr) / (rl + rr)
    a = torch.sqrt((GAMMA - 1) * (H - 0.5 * (u * u + v * v)))
    roe = (u, v, a, H)
    if name == "euler":
        b3 = (GAMMA - 1) / a ** 2 * ((H - u * u - v * v) * d[0] + u * d[mu] + v * d[mv] - d[3])
        b2 = d[mv] - v * d[0]
        b4 = (d[mu] + (a - u) * d[0] - a * b3) / (2 * a)
        b1 = d[0] - b3 - b4
        w = [_vec(4, {0: b1, mu: b1 * (u - a), mv: b1 * v, 3: b1 * (H - u * a)}),
             _vec(4, {0: b3, mu: b3 * u, mv: b3 * v, 3: b3 * 0.5 * (u * u + v * v)}),
             _vec(4, {mv: b2, 3: b2 * v}),
             _vec(4, {0: b4, mu: b4 * (u + a), mv: b4 * v, 3: b4 * (H + u * a)})]
        s = [u - a, u, u, u + a]

        def sound(q):
            return torch.sqrt(GAMMA * prim(q)[3] / q[0])

        m1, m4 = L + w[0], R - w[3]
        am, ap = _roe_split(s, w, ul - sound(L), m1[mu] / m1[0] - sound(m1), m4[mu] / m4[0] + sound(m4),
                            ur + sound(R), True)
        return w, s, am, ap, roe
    # the exact solver: states beside the contact, then the state at x/t = 0
    ps, us, side = _star(r_l, ul, pl, r_r, ur, pr)
    (rsl, s1, headl, taill), (rsr, s3, headr, tailr) = side

    def cons(r, un, ut, p):
        return _vec(4, {0: r, mu: r * un, mv: r * ut, 3: p / (GAMMA - 1) + 0.5 * r * (un * un + ut * ut)})

    def flux(r, un, ut, p):
        return _vec(4, {0: r * un, mu: r * un * un + p, mv: r * un * ut,
                        3: un * (p * GAMMA / (GAMMA - 1) + 0.5 * r * (un * un + ut * ut))})

    ql, qr = cons(rsl, us, vl, ps), cons(rsr, us, vr, ps)
    cl, cr = torch.sqrt(GAMMA * pl / r_l), torch.sqrt(GAMMA * pr / r_r)
    g = GAMMA
    left = us >= 0

    def sampled(sgn, r, un, p, c, rs, head, tail, shock):
        # mirrored so that the wave runs to the left: head <= tail (a shock: both its speed)
        cf = 2 / (g + 1) * (c + (g - 1) / 2 * sgn * un)
        rf, pf = r * (cf / c).clamp_min(1e-300) ** (2 / (g - 1)), p * (cf / c).clamp_min(1e-300) ** (2 * g / (g - 1))
        out = []
        for outside, inside, fan in ((r, rs, rf), (un, us, sgn * cf), (p, ps, pf)):
            x = torch.where(sgn * head >= 0, outside, torch.where(sgn * tail < 0, inside, fan))
            out.append(torch.where(shock, torch.where(sgn * head >= 0, outside, inside), x))
        return out

    lo = sampled(1.0, r_l, ul, pl, cl, rsl, headl, taill, ps > pl)
    hi = sampled(-1.0, r_r, ur, pr, cr, rsr, headr, tailr, ps > pr)
    r0, u0, p0 = (torch.where(left, x, y) for x, y in zip(lo, hi))
    f0 = flux(r0, u0, torch.where(left, vl, vr), p0)
    return [ql - L, qr - ql, R - qr], [s1, us, s3], f0 - flux(r_l, ul, vl, pl), flux(r_r, ur, vr, pr) - f0, roe


def _star(rl, ul, pl, rr, ur, pr):
    """p*, u* and, per side, (density, wave speed, head, tail) of the exact Euler Riemann problem (Toro, Riemann
    Solvers and Numerical Methods for Fluid Dynamics, ch. 4)."""
    g = GAMMA
    cl, cr = torch.sqrt(g * pl / rl), torch.sqrt(g * pr / rr)

    def f(p, r, pk, c):
        rare, shock = p / pk, torch.sqrt(2 / (g + 1) / r / (p + (g - 1) / (g + 1) * pk))
        a = 2 * c / (g - 1) * (rare ** ((g - 1) / (2 * g)) - 1)
        b = (p - pk) * shock
        da = rare ** (-(g + 1) / (2 * g)) / (r * c)
        db = (1 - 0.5 * (p - pk) / (p + (g - 1) / (g + 1) * pk)) * shock
        return torch.where(p <= pk, a, b), torch.where(p <= pk, da, db)

    z = (g - 1) / (2 * g)  # two rarefactions: a lower bound, from which Newton's steps rise
    p = ((cl + cr - 0.5 * (g - 1) * (ur - ul)).clamp_min(1e-12) / (cl / pl ** z + cr / pr ** z)) ** (1 / z)
    p = p.clamp_min(1e-12)  # (near vacuum the solver's tolerance stands in, there and for a negative step)
    for _ in range(60):
        (fl, dl), (fr, dr) = f(p, rl, pl, cl), f(p, rr, pr, cr)
        new = p - (fl + fr + ur - ul) / (dl + dr)
        new = torch.where(new < 0, 1e-12, new)
        moved = float((torch.abs(new - p) / new).max())
        p = new
        if moved < 4e-16:
            break
    same = (rl == rr) & (ul == ur) & (pl == pr)
    p = torch.where(same, pl, p)
    us = torch.where(same, ul, 0.5 * (ul + ur + f(p, rr, pr, cr)[0] - f(p, rl, pl, cl)[0]))
    sides = []
    for sgn, r, un, pk, c in ((1.0, rl, ul, pl, cl), (-1.0, rr, ur, pr, cr)):
        x = p / pk
        k = (g - 1) / (g + 1)
        rs = torch.where(p > pk, r * (x + k) / (k * x + 1), r * x ** (1 / g))
        cs = c * x ** z
        speed = un - sgn * c * torch.sqrt((g + 1) / (2 * g) * x + z)
        head, tail = un - sgn * c, us - sgn * cs
        sides.append((rs, torch.where(p > pk, speed, 0.5 * (head + tail)), torch.where(p > pk, speed, head), tail))
    return p, us, sides


def _rpt2(name, f, mu, roe, below, own, above):
    """Down- and up-going parts of a fluctuation f in the transverse direction."""
    mv = 3 - mu
    if name == "advection":
        s = 1.0 if mu == 1 else 0.5
        return min(s, 0.0) * f, max(s, 0.0) * f
    if name in ("acoustics", "vc_acoustics"):
        if name == "acoustics":
            cm = cp = math.sqrt(BULK / RHO)
            zm = z0 = zp = RHO * cm
        else:
            (rm, cm), (r0, c0), (rp, cp) = below, own, above
            zm, z0, zp = rm * cm, r0 * c0, rp * cp
        a1, a2 = (-f[0] + f[mv] * z0) / (zm + z0), (f[0] + f[mv] * z0) / (z0 + zp)
        return _vec(3, {0: cm * a1 * zm, mv: -cm * a1}), _vec(3, {0: cp * a2 * zp, mv: cp * a2})
    if name == "shallow":
        u, v, a = roe
        a1, a2, a3 = ((v + a) * f[0] - f[mv]) / (2 * a), f[mu] - u * f[0], (f[mv] - (v - a) * f[0]) / (2 * a)
        r = [(v - a, _vec(3, {0: a1, mu: a1 * u, mv: a1 * (v - a)})), (v, _vec(3, {mu: a2})),
             (v + a, _vec(3, {0: a3, mu: a3 * u, mv: a3 * (v + a)}))]
    else:
        u, v, a, H = roe
        b3 = (GAMMA - 1) / a ** 2 * ((H - u * u - v * v) * f[0] + u * f[mu] + v * f[mv] - f[3])
        b2 = f[mu] - u * f[0]
        b4 = (f[mv] + (a - v) * f[0] - a * b3) / (2 * a)
        b1 = f[0] - b3 - b4
        r = [(v - a, _vec(4, {0: b1, mu: b1 * u, mv: b1 * (v - a), 3: b1 * (H - v * a)})),
             (v, _vec(4, {0: b3, mu: b3 * u + b2, mv: b3 * v, 3: b3 * 0.5 * (u * u + v * v) + b2 * u})),
             (v + a, _vec(4, {0: b4, mu: b4 * u, mv: b4 * (v + a), 3: b4 * (H + v * a)}))]
    return sum(s.clamp_max(0) * w for s, w in r), sum(s.clamp_min(0) * w for s, w in r)


def _limiter(r, limiter):
    one, two = torch.ones_like(r), torch.full_like(r, 2.0)
    if limiter == "minmod":
        return torch.minimum(one, r).clamp_min(0)
    if limiter == "superbee":
        return torch.maximum(torch.minimum(one, 2 * r), torch.minimum(two, r)).clamp_min(0)
    if limiter == "vanleer":
        return (r + r.abs()) / (1 + r.abs())
    return torch.minimum((1 + r) / 2, torch.minimum(two, 2 * r)).clamp_min(0)


def _line(case, q, mu, ratio, aux):
    """Every interface 1 .. n+1 along the last axis of padded q: fluctuations, corrections, largest Courant
    number, transverse state."""
    name, n = case["solver"], q.shape[-1] - 4
    w, s, am, ap, roe = _rpn2(name, q[..., :-1], q[..., 1:], mu, *((aux[..., :-1], aux[..., 1:]) if aux is not None
                                                                   else (None, None)))
    cq = torch.zeros_like(am[..., 1:n + 2])
    top = 0.0
    for wk, sk in zip(w, s):
        mid, si = wk[..., 1:n + 2], sk[..., 1:n + 2]
        norm = (mid * mid).sum(0)
        dot = torch.where(si > 0, (wk[..., 0:n + 1] * mid).sum(0), (wk[..., 2:n + 3] * mid).sum(0))
        phi = torch.where(norm > 0, _limiter(dot / torch.where(norm > 0, norm, 1.0), case["limiter"]), 1.0)
        cq += si.abs() * (1 - si.abs() * ratio) * phi * mid
        top = max(top, float(si.abs().max()) * ratio)
    return am[..., 1:n + 2], ap[..., 1:n + 2], cq, top, tuple(x[..., 1:n + 2] for x in roe) if roe else None


def _step(case, q, aux, dt):
    """One step of padded q with its ghost cells filled: the interior and the Courant number."""
    (dx, dy), name = _spacing(case), case["solver"]
    lam, top = {1: dt / dx, 2: dt / dy}, 0.0

    def turned(a, mu):
        return a if mu == 1 or a is None else a.transpose(1, 2)

    if case["split"]:
        for mu in (1, 2):
            z = turned(q, mu)
            am, ap, cq, t, _ = _line(case, z, mu, lam[mu], turned(aux, mu))
            z = z.clone()
            z[..., 2:-2] -= lam[mu] * (ap - 0.5 * cq)[..., :-1] + lam[mu] * (am + 0.5 * cq)[..., 1:]
            q, top = turned(z, mu), max(top, t)
        return q[:, 2:-2, 2:-2], top
    dq = torch.zeros_like(q)
    for mu in (1, 2):
        z, d, x = turned(q, mu), turned(dq, mu), turned(aux, mu)
        J, n = z.shape[1], z.shape[2] - 4
        am, ap, cq, t, roe = _line(case, z[:, 1:J - 1], mu, lam[mu], x[:, 1:J - 1] if x is not None else None)
        top = max(top, t)
        h = 0.5 * lam[1] * lam[2]
        for f, c0, sgn in ((am, 1, 1.0), (ap, 2, -1.0)):  # what enters the left (c0 = 1) and the right cells
            cols = slice(c0, c0 + n + 1)
            d[:, 1:J - 1, cols] -= lam[mu] * (f + sgn * 0.5 * cq)
            if case["trans"] > 0:
                near = [x[:, k:J - 2 + k, cols] if x is not None else None for k in range(3)]
                down, up = _rpt2(name, f + sgn * cq if case["trans"] == 2 else f, mu, roe, *near)
                d[:, 1:J - 1, cols] += h * (up - down)
                d[:, 0:J - 2, cols] += h * down
                d[:, 2:J, cols] -= h * up
    return (q + dq)[:, 2:-2, 2:-2], top


def _exact_evolve(case, seed):
    q, aux = _initial(case, seed)
    auxbc = _fill(aux, case["bc"], 1.0) if aux is not None else None
    dt = _first_dt(case, q)
    t, tend, steps, cfl, first = 0.0, (case["steps"] - 0.5) * dt, 0, 0.0, True
    while t < tend:
        if not first:
            dt = dt * case["cfl"] / cfl
        first = False
        if t + dt > tend or tend - t - dt < 1e-14 * t:
            dt = tend - t
        new, cfl = _step(case, _fill(q, case["bc"]), auxbc, dt)
        if cfl <= (1.0 if case["cfl"] > 0.5 else 0.5):
            q, t, steps = new, t + dt, steps + 1
    return {"q": q, "t": t, "dt": dt, "cfl": cfl, "steps": steps}


def _exact_batch(case, seed):
    out = {"q": [], "t": [], "dt": [], "nsteps": [], "nreject": []}
    for side, (xs, ys), st, dt in _ensemble(case, seed):
        c = {"solver": "euler", "mx": side, "my": side, "split": False, "trans": 2, "limiter": "MC"}
        x, y = _centers(side, 0.0, 1.0)[None, :], _centers(side, 0.0, 1.0)[:, None]
        masks = {"NE": (x >= xs) & (y >= ys), "NW": (x < xs) & (y >= ys), "SW": (x < xs) & (y < ys),
                 "SE": (x >= xs) & (y < ys)}
        q = _euler_q(*(sum(m.double() * st[k][i] for k, m in masks.items()) for i in range(4)))
        t, done, rejected = 0.0, 0, 0
        for _ in range(case["steps"]):
            new, cfl = _step(c, _fill(q, "extrap"), None, dt)
            if not math.isfinite(float(new.sum())):
                break
            if cfl <= 1.0:
                q, t, done = new, t + dt, done + 1
            else:
                rejected += 1
            dt = dt * 0.9 / cfl
        out["q"].append(np.asfortranarray(_host(q)))
        for k, v in (("t", t), ("dt", dt), ("nsteps", done), ("nreject", rejected)):
            out[k].append(v)
    return {k: v if k == "q" else np.array(v, dtype=np.intc if k[0] == "n" else np.float64) for k, v in out.items()}


def _uniform(seed, i, k):
    """The sample generator's counter-based uniform numbers: splitmix64's finaliser, twice."""
    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    z = mix(np.uint64(seed) ^ mix(i * np.uint64(8) + np.uint64(k)))
    return torch.from_numpy((z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53).to(_device())


def _samples(seed, n):
    """Features, targets and validity of the training problems."""
    i = np.arange(n, dtype=np.uint64)
    with np.errstate(over="ignore"):
        U = [_uniform(int(seed), i, k) for k in range(6)]
    rl, pl, rr, pr = (torch.exp(math.log(10.0) * (-2.0 + 4.0 * U[k])) for k in (0, 1, 3, 4))
    ul, ur = -3.0 + 6.0 * U[2], -3.0 + 6.0 * U[5]
    g = GAMMA
    cl, cr = torch.sqrt(g * pl / rl), torch.sqrt(g * pr / rr)
    rb, pb = torch.sqrt(rl * rr), torch.sqrt(pl * pr)
    cb = torch.sqrt(g * pb / rb)
    x = torch.stack([0.5 * torch.log(rl / rr), 0.5 * torch.log(rr / rl), ul / cb, ur / cb, 0.5 * torch.log(pl / pr),
                     0.5 * torch.log(pr / pl)], 1)
    j2 = ((rr - rl) / rb) ** 2 + ((pr - pl) / pb) ** 2 + ((ur - ul) / cb) ** 2
    w = j2 / (1 + j2)
    ok = ~(2 / (g - 1) * (cl + cr) <= ur - ul)
    at = torch.nonzero(ok)[:, 0]
    rl, ul, pl, cl, rr, ur, pr, cr, w = (v[at] for v in (rl, ul, pl, cl, rr, ur, pr, cr, w))
    ps = _star(rl, ul, pl, rr, ur, pr)[0]
    # the adaptive guess: primitive-variable, two-rarefaction or two-shock (Toro, sec. 9.5.1)
    ppv = (0.5 * (pl + pr) + 0.125 * (ul - ur) * (rl + rr) * (cl + cr)).clamp_min(0.0)
    low, high = torch.minimum(pl, pr), torch.maximum(pl, pr)
    z = (g - 1) / (2 * g)
    pq = (pl / pr) ** z
    um = (pq * ul / cl + ur / cr + 2 / (g - 1) * (pq - 1)) / (pq / cl + 1 / cr)
    two = 0.5 * (pl * (1 + (g - 1) / 2 * (ul - um) / cl) ** (1 / z) + pr * (1 + (g - 1) / 2 * (um - ur) / cr) ** (1 / z))
    gl = torch.sqrt(2 / (g + 1) / rl / ((g - 1) / (g + 1) * pl + ppv))
    gr = torch.sqrt(2 / (g + 1) / rr / ((g - 1) / (g + 1) * pr + ppv))
    shock = (gl * pl + gr * pr - (ur - ul)) / (gl + gr)
    p0 = torch.where((high <= 2 * low) & (low <= ppv) & (ppv <= high), ppv, torch.where(ppv < low, two, shock))
    good = (p0 > 0) & (ps > 0)  # (a negative base above gives NaN: no guess)
    y = torch.zeros(n, dtype=torch.float64, device=x.device)
    y[at] = torch.where(good, torch.log(ps / p0.clamp_min(1e-300)) / w, 0.0)
    ok[at] = good
    return x.float().double(), y.float().double(), ok


def _exact_train(case, seed):
    x, y, ok = _samples(seed, case["samples"])
    p = torch.from_numpy(_weights(seed)).to(x.device).double()
    m, v, b, lr, loss, k = torch.zeros_like(p), torch.zeros_like(p), case["batch"], 3e-3, 0.0, 0
    count = case["samples"] // b
    for e in range(case["epochs"]):
        loss = torch.zeros((), dtype=torch.float64, device=x.device)
        for j in range(count):
            xs, ys, on = x[j * b:(j + 1) * b], y[j * b:(j + 1) * b], ok[j * b:(j + 1) * b].double()
            w1, b1, w2, b2, w3, b3 = (t.reshape(s) for t, s in zip(
                torch.split(p, [192, 32, 1024, 32, 32, 1]), [(32, 6), (32,), (32, 32), (32,), (32,), (1,)]))
            h1 = torch.tanh(xs @ w1.T + b1)
            h2 = torch.tanh(h1 @ w2.T + b2)
            err = on * (h2 @ w3 + b3 - ys)
            loss = loss + 0.5 * (err * err).sum() / b
            dy = err / b
            d2 = dy[:, None] * w3 * (1 - h2 * h2)
            d1 = (d2 @ w2) * (1 - h1 * h1)
            grad = torch.cat([(d1.T @ xs).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), h2.T @ dy,
                              dy.sum()[None]])
            k += 1
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            rate = lr * (1 - 0.9 * (e * count + j) / (case["epochs"] * count))
            p = p - rate * (m / (1 - 0.9 ** k)) / (torch.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
    return {"params": p, "loss": float(loss) / count}


def _exact_host(case, seed):
    q, _ = _initial(case, seed)
    new, cfl = _step(case, _fill(q, case["bc"], 1.0), None, _first_dt(case, q))
    return {"q": _host(new), "cfl": cfl}


def exact(case, seed):
    """What run() returns on its first pass, in 64 bits."""
    return {"evolve": _exact_evolve, "batch": _exact_batch, "train": _exact_train,
            "host": _exact_host}[case["kind"]](case, seed)

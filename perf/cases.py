"""Performance cases of the framework: what its users have it do, through its public entry points.

A case is a dict of plain values with a "kind":

* tube   -- a whole 1-D Riemann run (fill_riemann + Simulation.run), the reference's validation set-ups;
* step   -- the drop-in step a host calls once per time step (SplitSolver.solve, SplitSolver.max_wavespeed);
* loop   -- the device-resident 2-D / 3-D time loop (Simulation.run);
* batch  -- many independent 1-D / 2-D problems (Batch, its time loop captured once);
* adjoint -- a rollout and its gradient (adjoint.rollout under torch.autograd);
* levelset -- level-set advection and reinitialisation (LevelSetOps);
* bubble -- the two-material shock-bubble loop (MultiMaterial).

`exact` restates the schemes in plain torch, in 64 bits, from their definitions.
"""
import math
import random

import numpy as np
import torch

GAMMA = 1.4
DTYPES = {"f64": torch.float64, "f32": torch.float32}


def listed():
    return [
        # the reference's 1-D validation tubes: a few hundred cells, a few hundred steps; latency and launches
        {"name": "tube_f64_400", "kind": "tube", "nx": 400, "dtype": "f64", "flux": "hllc", "limiter": "vanleer",
         "walls": 0, "steps": 200},
        # a host program stepping a small, odd-sized grid itself, with the reference's default flux and limiter
        {"name": "step_f64_257x191", "kind": "step", "nx": 257, "ny": 191, "dtype": "f64", "flux": "force",
         "limiter": "superbee", "walls": 3, "steps": 4},
        # the benchmark's grid: four quadrants, FP64, HLLC
        {"name": "loop_f64_4096x4096", "kind": "loop", "nx": 4096, "ny": 4096, "nz": 1, "dtype": "f64", "flux": "hllc",
         "limiter": "vanleer", "walls": 0, "field": "riemann", "steps": 10},
        # an ordinary FP32 run on smooth flow
        {"name": "loop_f32_1920x1080", "kind": "loop", "nx": 1920, "ny": 1080, "nz": 1, "dtype": "f32", "flux": "hllc",
         "limiter": "vanleer", "walls": 0, "field": "smooth", "steps": 20},
        # an odd extent between walls, with FORCE
        {"name": "loop_f32_1001x750", "kind": "loop", "nx": 1001, "ny": 750, "nz": 1, "dtype": "f32", "flux": "force",
         "limiter": "vanleer", "walls": 3, "field": "smooth", "steps": 20},
        # the benchmark's 3-D variant: octants on 256^3
        {"name": "loop_f64_256x256x256", "kind": "loop", "nx": 256, "ny": 256, "nz": 256, "dtype": "f64",
         "flux": "hllc", "limiter": "vanleer", "walls": 0, "field": "riemann", "steps": 4},
        # a ragged 3-D box
        {"name": "loop_f32_150x131x97", "kind": "loop", "nx": 150, "ny": 131, "nz": 97, "dtype": "f32",
         "flux": "force", "limiter": "vanleer", "walls": 0, "field": "smooth", "steps": 10},
        # the batched workload: 3584 tubes and 512 quadrant problems
        {"name": "batch_f32_4096", "kind": "batch", "n1d": 3584, "n2d": 512, "lo1": 64, "hi1": 8192, "lo2": 64,
         "hi2": 512, "dtype": "f32", "flux": "hllc", "steps": 10},
        # the gradient workload's grid
        {"name": "adjoint_f64_1024x1024", "kind": "adjoint", "nx": 1024, "ny": 1024, "dtype": "f64", "flux": "hllc",
         "steps": 16},
        # a small ragged gradient in FP32
        {"name": "adjoint_f32_301x211", "kind": "adjoint", "nx": 301, "ny": 211, "dtype": "f32", "flux": "hllc",
         "steps": 9},
        # interface tracking on its own
        {"name": "levelset_1000x601", "kind": "levelset", "nx": 1000, "ny": 601},
        # the two-material benchmark: two reinitialisation cycles
        {"name": "bubble_f32_2048x1024", "kind": "bubble", "nx": 2048, "ny": 1024, "dtype": "f32", "flux": "hllc",
         "reinit_every": 5, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "step", "loop", "loop", "loop3", "batch", "adjoint", "levelset", "bubble"])
    dtype = rng.choice(["f64", "f32"])
    flux = rng.choice(["hllc", "hllc", "force"])
    limiter = rng.choice(["vanleer", "vanleer", "superbee"])
    if kind == "tube":
        return {"kind": kind, "nx": _log(rng, 100, 8000), "dtype": dtype, "flux": flux, "limiter": limiter,
                "walls": rng.choice([0, 0, 1]), "steps": rng.randint(100, 300)}
    if kind == "step":
        return {"kind": kind, "nx": _log(rng, 64, 1500), "ny": _log(rng, 64, 1500), "dtype": dtype, "flux": flux,
                "limiter": limiter, "walls": rng.choice([0, 0, 1, 2, 3]), "steps": rng.randint(2, 6)}
    if kind == "loop":
        nx, ny = _log(rng, 100, 3000), _log(rng, 100, 3000)
        if rng.random() < 0.5:      # half of them in the multiples of eight that users tend to pick
            nx, ny = (nx + 7) // 8 * 8, (ny + 7) // 8 * 8
        return {"kind": kind, "nx": nx, "ny": ny, "nz": 1, "dtype": dtype, "flux": flux, "limiter": limiter,
                "walls": rng.choice([0, 0, 1, 2, 3]), "field": rng.choice(["riemann", "smooth"]),
                "steps": rng.randint(5, 20)}
    if kind == "loop3":
        n = [_log(rng, 40, 220) for _ in range(3)]
        return {"kind": "loop", "nx": n[0], "ny": n[1], "nz": n[2], "dtype": dtype, "flux": flux, "limiter": "vanleer",
                "walls": rng.choice([0, 0, 5, 7]), "field": rng.choice(["riemann", "smooth"]),
                "steps": rng.randint(2, 6)}
    if kind == "batch":
        return {"kind": kind, "n1d": _log(rng, 16, 1500), "n2d": _log(rng, 4, 150), "lo1": 64,
                "hi1": rng.choice([1000, 4000]), "lo2": 64, "hi2": rng.choice([200, 400]), "dtype": dtype,
                "flux": flux, "steps": rng.randint(5, 20)}
    if kind == "adjoint":
        return {"kind": kind, "nx": _log(rng, 100, 900), "ny": _log(rng, 100, 900), "dtype": dtype, "flux": flux,
                "steps": rng.randint(4, 16)}
    if kind == "levelset":
        return {"kind": kind, "nx": _log(rng, 150, 2000), "ny": _log(rng, 150, 1200)}
    nx = _log(rng, 200, 1600)
    return {"kind": "bubble", "nx": nx, "ny": max(100, nx // 2 + rng.randint(-30, 30)), "dtype": dtype, "flux": "hllc",
            "reinit_every": rng.choice([2, 5]), "steps": rng.randint(3, 8)}


# ---- shapes and inputs -------------------------------------------------------------------------------------------

def _shape(case):
    n = [case["nx"]]
    if case["kind"] != "tube":
        n.append(case["ny"])
    if case.get("nz", 1) > 1:
        n.append(case["nz"])
    return tuple(n)


def _orthants(seed, dims):
    """2**dims primitive states (rho, p, v...): moderate shock-tube ratios, as in the reference's Toro and Liska
    validation cases (the strongest of those need a lower CFL number than the loop's)."""
    r = random.Random("%d/orthants" % seed)
    out = np.zeros((2 ** dims, dims + 2))
    for s in out:
        s[0] = math.exp(r.uniform(math.log(0.25), math.log(2.0)))
        s[1] = math.exp(r.uniform(math.log(0.2), math.log(2.5)))
        s[2:] = [r.uniform(-0.7, 0.7) for _ in range(dims)]
    return out


def _smooth(seed, shape, device):
    """A smooth random conservative state (dims + 2, cells) in 64 bits, x fastest: low sine modes plus a steep front
    that turns into a shock."""
    r = random.Random("%d/smooth" % seed)
    dims = len(shape)
    axes = [(torch.arange(n, device=device, dtype=torch.float64) + 0.5) / n for n in shape]

    def field():
        f = torch.zeros(shape[::-1], device=device, dtype=torch.float64)
        for _ in range(4):
            g = torch.full((1,) * dims, r.uniform(0.5, 1.0), device=device, dtype=torch.float64)
            for d, x in enumerate(axes):
                k, ph = r.randint(1, 4), r.uniform(0, 2 * math.pi)
                g = g * torch.sin(2 * math.pi * k * x + ph).view([-1 if a == dims - 1 - d else 1 for a in range(dims)])
            f = f + g
        return f / 4

    c = r.uniform(0.35, 0.65)
    front = torch.tanh((axes[0] - c) * shape[0] / 6.0)          # about six cells wide
    rho = torch.exp(0.5 * field()) * (1.3 - 0.3 * front)
    p = torch.exp(0.4 * field()) * (1.6 - 0.6 * front)
    v = [0.5 * field() for _ in range(dims)]
    energy = p / (GAMMA - 1) + 0.5 * rho * sum(w * w for w in v)
    return torch.stack([rho, energy] + [rho * w for w in v]).reshape(dims + 2, -1)


def _distance(seed, nx, ny, h, device):
    """A level set: two bubbles and a ripple, no signed distance away from its zero line (reinitialisation's work)."""
    r = random.Random("%d/bubbles" % seed)
    x = (torch.arange(nx, device=device, dtype=torch.float64) + 0.5) * h
    y = ((torch.arange(ny, device=device, dtype=torch.float64) + 0.5) * h).view(-1, 1)
    w, t = nx * h, ny * h
    f = None
    for k in range(2):
        cx, cy, rad = w * r.uniform(0.2 + 0.4 * k, 0.35 + 0.4 * k), t * r.uniform(0.4, 0.6), min(w, t) * r.uniform(0.1, 0.2)
        g = torch.sqrt((x - cx) ** 2 + (y - cy) ** 2) - rad
        f = g if f is None else torch.minimum(f, g)
    f = f * (1.0 + 0.2 * torch.sin(7.0 * x / w + r.uniform(0, 6)) * torch.sin(5.0 * y / t + r.uniform(0, 6)))
    vel = 0.6 * torch.sin(4.0 * x / w + r.uniform(0, 6)) * torch.cos(3.0 * y / t + r.uniform(0, 6)) + 0.1
    return f.reshape(-1).contiguous(), vel.expand(ny, nx).reshape(-1).contiguous()


def _problems(case, seed):
    """The case's problem sizes (the same for every seed) with the seed's states."""
    sizes, r = random.Random("sizes"), random.Random("%d/batch" % seed)
    out = []
    for i in range(case["n1d"] + case["n2d"]):
        if i < case["n1d"]:
            shape = (_log(sizes, case["lo1"], case["hi1"]),)
        else:
            s = _log(sizes, case["lo2"], case["hi2"])
            shape = (s, s)
        out.append((shape, _orthants(r.randrange(1 << 30), len(shape))))
    return out


def _bubble_spec(case, seed):
    from fluidity_b200.workloads import shock_bubble
    return shock_bubble(seed % (1 << 31), case["nx"], case["ny"])


def _cotangent(seed, shape, device):
    """A smooth gradient of some objective with respect to the final state."""
    return _smooth(seed + 7919, shape, device) - 1.0


CFL = {"tube": 0.9, "loop": 0.8, "batch": 0.8, "adjoint": 0.7, "bubble": 0.6}


def _step_dtdh(state, shape):
    """dt/dh of CFL 0.6 on the step case's initial state, with room for what the flow does in a few steps."""
    return 0.6 / float(_wavespeed(_planes(state.double(), shape)))


def prepare(case, seed):
    from fluidity_b200.adjoint import Adjoint
    from fluidity_b200.batch import Batch
    from fluidity_b200.levelset import LevelSetOps
    from fluidity_b200.multimaterial import MultiMaterial
    from fluidity_b200.solver import Simulation, SplitSolver
    kind, dev = case["kind"], torch.device("cuda")
    s = {"case": case}
    if kind in ("tube", "step", "loop"):
        shape = _shape(case)
        s["solver"] = SplitSolver(shape, dtype=case["dtype"], flux=case["flux"], limiter=case["limiter"], gamma=GAMMA,
                                  boundary_mask=case["walls"])
        s["a"], s["b"] = s["solver"].new_state(), s["solver"].new_state()
        if kind == "tube" or case.get("field") == "riemann":
            s["states"] = _orthants(seed, len(shape))
        else:
            s["u0"] = _smooth(seed, shape, dev).to(DTYPES[case["dtype"]])
        if kind == "step":
            s["dtdh"] = _step_dtdh(s["u0"], shape)
            s["ws"] = torch.empty(1, dtype=torch.float64, device=dev)
        else:
            s["sim"] = Simulation(s["solver"])
    elif kind == "batch":
        b = Batch(_problems(case, seed), dtype=case["dtype"], flux=case["flux"], gamma=GAMMA)
        b.fill()
        s["batch"], s["a0"] = b, b.a.clone()
        b.begin(CFL[kind], 1e30, case["steps"])
        b.capture(case["steps"])
    elif kind == "adjoint":
        shape = _shape(case)
        s["adj"] = Adjoint(shape, case["steps"], dtype=case["dtype"], flux=case["flux"], gamma=GAMMA)
        s["u0"] = _smooth(seed, shape, dev).to(DTYPES[case["dtype"]]).requires_grad_(True)
        s["lam"] = _cotangent(seed, shape, dev).to(DTYPES[case["dtype"]])
    elif kind == "levelset":
        h = 1.0 / case["nx"]
        s["ops"], s["h"] = LevelSetOps((case["nx"], case["ny"])), h
        s["phi"], s["vel"] = _distance(seed, case["nx"], case["ny"], h, dev)
        s["moved"], s["out"] = s["ops"].new(), s["ops"].new()
    else:
        mm = MultiMaterial.shock_bubble(_bubble_spec(case, seed), dtype=case["dtype"], flux=case["flux"])
        s["mm"] = mm
        s["keep"] = [(t, t.clone()) for t in (mm.u[0][0], mm.u[1][0], mm.phi[0][0], mm.phi[1][0])]
    return s


def run(s):
    from fluidity_b200.adjoint import rollout
    case = s["case"]
    kind = case["kind"]
    if kind in ("tube", "loop"):
        if "states" in s:
            s["solver"].fill_riemann(s["states"], out=s["a"])
        else:
            s["a"].copy_(s["u0"])
        state, iters, t = s["sim"].run(s["a"], s["b"], CFL[kind], 1.0 / case["nx"], 1e30, case["steps"])
        return {"state": state, "iters": iters, "time": t}
    if kind == "step":
        a, b = s["a"], s["b"]
        a.copy_(s["u0"])
        for _ in range(case["steps"]):
            a, b = s["solver"].solve(a, b, s["dtdh"], max_ws=s["ws"])
            a, b = b, a            # the new state is the next step's input
        return {"state": a, "wavespeed": s["ws"]}
    if kind == "batch":
        b = s["batch"]
        b.a.copy_(s["a0"])
        b.begin(CFL[kind], 1e30, case["steps"])
        b.launch()
        return {"arena": b.a}
    if kind == "adjoint":
        u = rollout(s["u0"], s["adj"], CFL[kind], 1.0 / case["nx"])
        (grad,) = torch.autograd.grad(u, s["u0"], s["lam"])
        return {"state": u.detach(), "gradient": grad}
    if kind == "levelset":
        s["ops"].advect(s["phi"], s["vel"], 0.5 * s["h"], s["h"], out=s["moved"])
        s["ops"].reinit(s["moved"], s["h"], out=s["out"])
        return {"advected": s["moved"], "distance": s["out"]}
    mm = s["mm"]
    for t, v in s["keep"]:
        t.copy_(v)
    mm.begin(CFL[kind], 1e30, case["steps"], case["reinit_every"])
    mm.steps(case["steps"])
    phi = mm.current_phi()
    u = mm.states()
    return {"u0": u[0], "u1": u[1], "phi0": phi[0], "phi1": phi[1]}


# ---- work and tolerances -----------------------------------------------------------------------------------------

def work(case):
    """Each time step reads and writes the state once; the arithmetic of a cell is counted from the scheme (about 300
    operations per cell and sweep, four times that for a sweep's reverse)."""
    kind, size = case["kind"], 8 if case.get("dtype", "f64") == "f64" else 4
    if kind in ("tube", "step", "loop"):
        shape = _shape(case)
        d, cells = len(shape), math.prod(shape)
        return {"bytes": 2 * (d + 2) * size * cells * case["steps"], "flops": 300 * d * cells * case["steps"]}
    if kind == "batch":
        def mean(lo, hi, p):   # of n**p, n log-uniform
            return (hi ** p - lo ** p) / (p * math.log(hi / lo))
        one, two = case["n1d"] * mean(case["lo1"], case["hi1"], 1), case["n2d"] * mean(case["lo2"], case["hi2"], 2)
        return {"bytes": (2 * 3 * one + 2 * 4 * two) * size * case["steps"],
                "flops": 300 * (one + 2 * two) * case["steps"]}
    cells = case["nx"] * case["ny"]
    if kind == "adjoint":   # forward: state in and out; backward: state and adjoint in, adjoint out
        return {"bytes": 5 * 4 * size * cells * case["steps"], "flops": 300 * 2 * 5 * cells * case["steps"]}
    if kind == "levelset":  # advection: phi, velocity in, phi out (three stages); reinitialisation: in and out
        return {"bytes": (3 * 3 * 8 + 2 * 8) * cells, "flops": (3 * 160 + 60) * cells}
    per = 2 * 2 * 4 * size + 2 * 3 * 3 * 8 + 2 * 2 * 8 / case["reinit_every"]
    return {"bytes": per * cells * case["steps"], "flops": (2 * 2 * 300 + 2 * 3 * 160) * cells * case["steps"]}


def tolerance(case):
    """Against `exact`, FP64 runs were measured at 1e-16 to 9e-16, FP32 runs at 6e-8 to 1.3e-7 and the FP32 bubble at
    8e-8.  Sums in another order grow like those errors with the step count and fall on either side of a wave, limiter
    or flattening test now and then, which moves a value by more than its rounding; a gradient feels such a switch most
    (measured at 1.2e-4 and 2.8e-4 in FP32, 6e-16 in FP64 where no test fell differently)."""
    kind = case["kind"]
    f64 = case.get("dtype", "f64") == "f64"
    if kind == "levelset":
        return {"rel": 1e-13}
    if kind == "adjoint":
        return {"rel": 1e-9} if f64 else {"rel": 2e-3, "max": 0.5}
    if kind == "bubble":
        return {"rel": 1e-10} if f64 else {"rel": 2e-6}
    return {"rel": 1e-12} if f64 else {"rel": 2e-6}


# ---- 64-bit restatement ------------------------------------------------------------------------------------------
#
# States are (dims + 2, nz, ny, nx) or with fewer axes; dimension d is axis -(d + 1).

def _planes(u, shape):
    return u[:, :math.prod(shape)].reshape((-1,) + tuple(shape[::-1]))


def _pressure(u):
    return (GAMMA - 1) * (u[1] - 0.5 * sum(m * m for m in u[2:]) / u[0])


def _wavespeed(u):
    v = torch.stack([(m / u[0]).abs() for m in u[2:]]).amax(0)
    return (v + torch.sqrt(GAMMA * _pressure(u) / u[0])).max()


def _mirror(u, walls, g):
    """g mirror ghosts on every side; a wall (bit d of walls) negates the normal momentum."""
    dims = u.dim() - 1
    for d in range(dims):
        ax = u.dim() - 1 - d
        n = u.shape[ax]
        lo, hi = u.narrow(ax, 0, g).flip(ax), u.narrow(ax, n - g, g).flip(ax)
        if (walls >> d) & 1:
            sign = torch.ones([dims + 2] + [1] * dims, dtype=u.dtype, device=u.device)
            sign[2 + d] = -1
            lo, hi = lo * sign, hi * sign
        u = torch.cat([lo, u, hi], ax)
    return u


def _at(f, k, d):
    """f at index + k along dimension d (edges wrap; the ghosts keep that away from the cells that count)."""
    return torch.roll(f, -k, f.dim() - 1 - d)


def _min(a, b):
    return torch.where(b < a, b, a)


def _flat(p, v, d):
    """The flattening coefficient's base along d: 1, or its ramp where the flow is a steep compression."""
    pn, pp = _at(p, 1, d), _at(p, -1, d)
    dp = (pn - pp).abs()
    on = (_at(v, -1, d) - _at(v, 1, d) > 0) & (dp > 0.33 * _min(pn, pp))
    wide = (_at(p, 2, d) - _at(p, -2, d)).abs()
    eta = 1 - (dp / torch.where(on & (wide > 0), wide, 1.0) - 0.75) / 0.1
    eta = torch.where(wide > 0, eta, 0.0)
    eta = torch.where(eta > 0, eta, 0.0)
    eta = torch.where(eta < 1, eta, 1.0)
    return torch.where(on, eta, 1.0)


def _limited(bd, fd, limiter):
    if limiter == "superbee":
        safe = torch.where(fd == 0, 1.0, fd)
        r = bd / safe
        er = 2 / (1 + torch.where(r > 0, r, 1.0))
        xi = torch.where(r <= 0.5, 2 * r, torch.where(r <= 1, torch.ones_like(r), _min(_min(r, er), torch.full_like(r, 2.0))))
        return torch.where((r <= 0) | (fd == 0), 0.0, 0.5 * (bd + fd) * xi)
    # van Leer as the framework has it, 0.5 (bd + fd) 2 min(r, 1) / (1 + r): minmod
    return torch.where(bd * fd > 0, torch.where(bd.abs() <= fd.abs(), bd, fd), 0.0)


def _flux(u, d):
    v, p = u[2 + d] / u[0], _pressure(u)
    f = [u[2 + d], v * (u[1] + p)] + [m * v for m in u[2:]]
    f[2 + d] = f[2 + d] + p
    return torch.stack(f)


def _hllc(l, r, d):
    pl, pr, vl, vr = _pressure(l), _pressure(r), l[2 + d] / l[0], r[2 + d] / r[0]
    al, ar = torch.sqrt(GAMMA * pl / l[0]), torch.sqrt(GAMMA * pr / r[0])
    ps = 0.5 * ((pl + pr) - 0.25 * (vr - vl) * (r[0] + l[0]) * (al + ar))
    ps = torch.where(ps > 0, ps, 0.0)
    q = (GAMMA + 1) / (2 * GAMMA)
    sl = torch.where(ps <= pl, vl - al, vl - al * torch.sqrt(1 + q * (ps / pl - 1)))
    sr = torch.where(ps <= pr, vr + ar, vr + ar * torch.sqrt(1 + q * (ps / pr - 1)))
    ml, mr = l[0] * (sl - vl), r[0] * (sr - vr)
    sm = (pr - pl + vl * ml - vr * mr) / (ml - mr)

    def side(u, s, v, p):
        c = (s - v) / (s - sm)
        st = [c * w for w in u]
        st[2 + d] = sm * u[0] * c
        st[1] = c * (u[1] + u[0] * (sm - v) * (sm + p / (u[0] * (s - v))))
        return _flux(u, d) + s * (torch.stack(st) - u)

    f = torch.where(sm >= 0, side(l, sl, vl, pl), side(r, sr, vr, pr))
    f = torch.where(sr <= 0, _flux(r, d), f)
    return torch.where(sl >= 0, _flux(l, d), f)


def _force(l, r, d, dtdh):
    fl, fr = _flux(l, d), _flux(r, d)
    lf = 0.5 * (fl + fr + (l - r) / dtdh)
    return 0.5 * (lf + _flux(0.5 * (l + r + dtdh * (fl - fr)), d))


def _sweep(u, d, dtdh, case):
    """One dimensional sweep: MUSCL-Hancock with flattening, the Riemann flux, the conservative update."""
    dims, g = u.dim() - 1, 4
    w = _mirror(u, case.get("walls", 0), g)
    p = _pressure(w)
    chi = None
    for e in range(dims):
        base = _flat(p, w[2 + e] / w[0], e)
        rise = _at(p, 1, e) - _at(p, -1, e)
        c = _min(base, torch.where(rise > 0, _at(base, 1, e), torch.where(rise < 0, _at(base, -1, e), base)))
        chi = c if chi is None else _min(chi, c)
    half = 0.5 * chi * _limited(w - _at(w, -1, d), _at(w, 1, d) - w, case.get("limiter", "vanleer"))
    lo, hi = w - half, w + half
    df = 0.5 * dtdh * (_flux(lo, d) - _flux(hi, d))
    left, right = _at(hi + df, -1, d), lo + df          # the two states at the face below each cell
    # cells whose stencils reach past the ghosts hold wrapped values: cut them before the Riemann solve
    for e in range(dims):
        ax = left.dim() - 1 - e
        n = left.shape[ax] - 2 * g
        left, right = (t.narrow(ax, g, n + (1 if e == d else 0)) for t in (left, right))
    f = _hllc(left, right, d) if case["flux"] == "hllc" else _force(left, right, d, dtdh)
    ax = u.dim() - 1 - d
    n = u.shape[ax]
    return u + dtdh * (f.narrow(ax, 0, n) - f.narrow(ax, 1, n))


def _run(u, case, cfl, dh, steps):
    t = 0.0
    for _ in range(steps):
        dt = cfl * dh / _wavespeed(u)
        for d in range(u.dim() - 1):
            u = _sweep(u, d, dt / dh, case)
        t = t + dt
    return u, float(t)


def _riemann(shape, states, device):
    dims = len(shape)
    which = torch.zeros(shape[::-1], dtype=torch.int64, device=device)
    for d, n in enumerate(shape):
        x = torch.from_numpy(~(np.arange(n, dtype=np.float32) / np.float32(n) < 0.5)).to(device)
        which = which + (x.long() << d).view([-1 if a == dims - 1 - d else 1 for a in range(dims)])
    s = torch.from_numpy(states).to(device)
    cons = torch.stack([s[:, 0], s[:, 1] / (GAMMA - 1) + 0.5 * s[:, 0] * (s[:, 2:] ** 2).sum(1)] +
                       [s[:, 0] * s[:, 2 + d] for d in range(dims)])
    return cons[:, which]


def _reinit_exact(phi, h):
    """Sources keep |phi|; the rest is the fixed point of the Godunov eikonal solve, by Jacobi iteration."""
    big = 1e300

    def near(f, fill):
        q = torch.full((f.shape[0] + 2, f.shape[1] + 2), fill, dtype=f.dtype, device=f.device) if fill is not None else \
            _mirror(f.unsqueeze(0), 0, 1)[0]
        if fill is not None:
            q[1:-1, 1:-1] = f
        return q[1:-1, :-2], q[1:-1, 2:], q[:-2, 1:-1], q[2:, 1:-1]

    fixed = torch.zeros_like(phi, dtype=torch.bool)
    for o in near(phi, None):
        fixed |= (torch.sign(phi) != torch.sign(o)) & (phi.abs() < o.abs())
    u = torch.where(fixed, phi.abs(), big)
    for k in range(1, 100000):
        xm, xp, ym, yp = near(u, big)
        a, b = torch.minimum(xm, xp), torch.minimum(ym, yp)
        apart = (a - b).abs() >= h
        q = torch.where(apart, torch.minimum(a, b) + h,
                        0.5 * (a + b + torch.sqrt(2 * h * h - torch.where(apart, 0.0, a - b) ** 2)))
        new = torch.where(fixed, u, torch.minimum(u, q))
        if k % 64 == 0 and torch.equal(new, u):
            break
        u = new
    return torch.sign(phi) * u


def _weno(d1, d2, d3, d4, d5):
    sq = torch.stack([d1 * d1, d2 * d2, d3 * d3, d4 * d4, d5 * d5]).amax(0)
    eps = 1e-5 * sq + 1e-98
    b = [13 / 12 * (d1 - 2 * d2 + d3) ** 2 + 0.25 * (d1 - 4 * d2 + 3 * d3) ** 2,
         13 / 12 * (d2 - 2 * d3 + d4) ** 2 + 0.25 * (d2 - d4) ** 2,
         13 / 12 * (d3 - 2 * d4 + d5) ** 2 + 0.25 * (3 * d3 - 4 * d4 + d5) ** 2]
    w = [c / ((s + eps) / eps) ** 2 for c, s in zip((0.1, 0.6, 0.3), b)]
    v = [(2 * d1 - 7 * d2 + 11 * d3) / 6, (-d2 + 5 * d3 + 2 * d4) / 6, (2 * d3 + 5 * d4 - d5) / 6]
    return sum(x * y for x, y in zip(w, v)) / sum(w)


def _advect_exact(phi, vel, dt, h):
    def ham(f):
        q = _mirror(f.unsqueeze(0), 0, 3)[0]
        r = torch.zeros_like(f)
        for d in range(2):
            e = [(_at(q, k + 1, d) - _at(q, k, d)) / h for k in range(-3, 3)]
            back = _weno(e[0], e[1], e[2], e[3], e[4])[3:-3, 3:-3]
            ahead = _weno(e[5], e[4], e[3], e[2], e[1])[3:-3, 3:-3]
            neg = vel <= 0
            b = torch.where(neg, back.clamp(min=0), back.clamp(max=0))
            a = torch.where(neg, ahead.clamp(max=0), ahead.clamp(min=0))
            r = r + torch.maximum(b * b, a * a)
        return vel * torch.sqrt(r)

    s = phi - dt * ham(phi)
    s = 0.75 * phi + 0.25 * (s - dt * ham(s))
    return phi / 3 + 2 / 3 * (s - dt * ham(s))


def _adjoint_exact(case, seed, device):
    from torch.utils.checkpoint import checkpoint
    shape = _shape(case)
    u0 = _planes(_smooth(seed, shape, device).to(DTYPES[case["dtype"]]).double(), shape).requires_grad_(True)
    lam = _planes(_cotangent(seed, shape, device).to(DTYPES[case["dtype"]]).double(), shape)

    def sweep(u, d, dtdh):
        return _sweep(u, d, dtdh, case)

    u = u0
    for _ in range(case["steps"]):
        dtdh = CFL["adjoint"] / float(_wavespeed(u.detach()))
        for d in range(2):
            u = checkpoint(sweep, u, d, dtdh, use_reentrant=False)
    (g,) = torch.autograd.grad(u, u0, lam)
    return {"state": u.detach().reshape(4, -1), "gradient": g.reshape(4, -1)}


def exact(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    if kind in ("tube", "loop"):
        shape = _shape(case)
        if kind == "tube" or case["field"] == "riemann":
            u = _riemann(shape, _orthants(seed, len(shape)), dev)
        else:
            u = _planes(_smooth(seed, shape, dev).to(DTYPES[case["dtype"]]).double(), shape)
        u, t = _run(u, case, CFL[kind], 1.0 / case["nx"], case["steps"])
        return {"state": u.reshape(len(shape) + 2, -1), "iters": case["steps"], "time": t}
    if kind == "step":
        shape = _shape(case)
        u0 = _smooth(seed, shape, dev).to(DTYPES[case["dtype"]])
        dtdh, u = _step_dtdh(u0, shape), _planes(u0.double(), shape)
        for _ in range(case["steps"]):
            for d in range(2):
                u = _sweep(u, d, dtdh, case)
        return {"state": u.reshape(4, -1), "wavespeed": _wavespeed(u).reshape(1)}
    if kind == "batch":
        problems = _problems(case, seed)
        if len(problems) > 100:      # one problem at a time: minutes for thousands
            return None
        parts = []
        for shape, states in problems:
            u, _ = _run(_riemann(shape, states, dev), case, CFL[kind], 1.0 / shape[0], case["steps"])
            cells = math.prod(shape)
            plane = torch.zeros(len(shape) + 2, (cells + 31) // 32 * 32, dtype=torch.float64, device=dev)
            plane[:, :cells] = u.reshape(len(shape) + 2, -1)
            parts.append(plane.reshape(-1))
        return {"arena": torch.cat(parts)}
    if kind == "adjoint":
        return _adjoint_exact(case, seed, dev)
    if kind == "levelset":
        h = 1.0 / case["nx"]
        phi, vel = _distance(seed, case["nx"], case["ny"], h, dev)
        moved = _advect_exact(phi.view(case["ny"], -1), vel.view(case["ny"], -1), 0.5 * h, h)
        return {"advected": moved.reshape(-1), "distance": _reinit_exact(moved, h).reshape(-1)}
    return _bubble_exact(case, seed, dev)


# ---- the two-material step ---------------------------------------------------------------------------------------

def _bubble_exact(case, seed, dev):
    spec = _bubble_spec(case, seed)
    nx, ny, h, gam = case["nx"], case["ny"], spec["h"], spec["gammas"]

    def gas(prim, g):
        e = prim[1] / (g - 1) + 0.5 * prim[0] * (prim[2] ** 2 + prim[3] ** 2)
        c = torch.tensor([prim[0], e, prim[0] * prim[2], prim[0] * prim[3]], dtype=torch.float64, device=dev)
        return c.view(4, 1, 1).expand(4, ny, nx)

    behind = torch.from_numpy(spec["shock_phi"]).to(dev).view(ny, nx) <= 0
    u = [torch.where(behind, gas(spec["shocked"], gam[0]), gas(spec["ambient"], gam[0])),
         gas(spec["bubble"], gam[1]).clone()]
    if case["dtype"] == "f32":
        u = [x.float().double() for x in u]
    phi = [torch.from_numpy(spec[k]).to(dev).view(ny, nx) for k in ("phi0", "phi1")]
    for it in range(case["steps"]):
        u = _ghosts(u, phi, h, gam)
        speed = max(float(_with_gamma(g, _wavespeed, x)) for g, x in zip(gam, u))
        dt = CFL["bubble"] * h / speed
        for d in range(2):
            u = [_with_gamma(g, _sweep, x, d, dt / h, {"flux": case["flux"]}) for g, x in zip(gam, u)]
        vel = torch.zeros_like(phi[0])
        for x, f in reversed(list(zip(u, phi))):
            q = _mirror(f.unsqueeze(0), 0, 1)[0]
            gx, gy = (q[1:-1, 2:] - q[1:-1, :-2]) / (2 * h), (q[2:, 1:-1] - q[:-2, 1:-1]) / (2 * h)
            vel = torch.where(f <= 0, (x[2] * gx + x[3] * gy) / (x[0] * torch.sqrt(gx * gx + gy * gy)), vel)
        a, b = (_advect_exact(f, vel, dt, h) for f in phi)
        a = a - 0.5 * (a + b)
        if (it + 1) % case["reinit_every"] == 0:
            a = _reinit_exact(a, h)
        phi = [a, -a]
    return {"u0": u[0].reshape(4, -1), "u1": u[1].reshape(4, -1), "phi0": phi[0].reshape(-1), "phi1": phi[1].reshape(-1)}


def _with_gamma(g, f, *args):
    global GAMMA
    keep, GAMMA = GAMMA, g
    try:
        return f(*args)
    finally:
        GAMMA = keep


def _ghosts(u, phi, h, gam):
    """Riemann ghost-fluid star states next to the interface, then extrapolation through a band of ghost cells."""
    return [_extrapolate(_star_cells(u[m], u[1 - m], phi[m], phi[1 - m], h, gam[m], gam[1 - m]), phi[m], h)
            for m in range(2)]


def _star_cells(ua, ub, pa, pb, h, ga, gb):
    ny, nx = pa.shape
    q = _mirror(pa.unsqueeze(0), 0, 1)[0]
    xm, xp, ym, yp = q[1:-1, :-2], q[1:-1, 2:], q[:-2, 1:-1], q[2:, 1:-1]
    gx, gy = 0.5 * (xp - xm), 0.5 * (yp - ym)
    s = torch.sqrt(gx * gx + gy * gy)
    src = (pa <= 0) & (pa >= -h) & (xm != 0) & (xp != 0) & (ym != 0) & (yp != 0) & (pb >= 0) & (pb < h) & (s > 0)
    y, x = torch.nonzero(src, as_tuple=True)
    n = torch.stack([gx[y, x], gy[y, x]]) / s[y, x]
    far = pa[y, x].abs()

    def clip(i, k):
        i = torch.where(i < 0, -1 - i, torch.where(i >= k, 2 * k - 1 - i, i))
        return i.clamp(0, k - 1)

    def probe(u, w):
        sg, off = torch.sign(w).long(), w.abs().floor()
        f = w.abs() - off
        o = (torch.sign(w) * off).long()
        x0, x1 = u[:, y, clip(x + o[0], nx)], u[:, y, clip(x + o[0] + sg[0], nx)]
        y0, y1 = u[:, clip(y + o[1], ny), x], u[:, clip(y + o[1] + sg[1], ny), x]
        return (x0 * (1 - f[0]) + x1 * f[0]) * (1 - f[1]) + (y0 * (1 - f[0]) + y1 * f[0]) * f[1]

    l, r = probe(ua, n * (far - 1.5 * h) / h), probe(ub, n * (far + 1.5 * h) / h)
    vl, vr = l[2:] / l[0], r[2:] / r[0]
    vln, vrn = (vl * n).sum(0), (vr * n).sum(0)
    l, r = (torch.stack([w[0], w[1], v * w[0], 0 * w[0]]) for w, v in ((l, vln), (r, vrn)))
    pl, pr = _with_gamma(ga, _pressure, l), _with_gamma(gb, _pressure, r)
    al, ar = torch.sqrt(ga * pl / l[0]), torch.sqrt(gb * pr / r[0])
    ps = (0.5 * ((pl + pr) - 0.25 * (vrn - vln) * (r[0] + l[0]) * (al + ar))).clamp(min=0)
    sl = vln - al * torch.where(ps <= pl, 1.0, torch.sqrt((1 + (ga + 1) / (2 * ga) * (ps / pl - 1)).clamp(min=0)))
    sr = vrn + ar * torch.where(ps <= pr, 1.0, torch.sqrt((1 + (gb + 1) / (2 * gb) * (ps / pr - 1)).clamp(min=0)))
    ml, mr = l[0] * (sl - vln), r[0] * (sr - vrn)
    sm = (pr - pl + vln * ml - vrn * mr) / (ml - mr)
    c = (sl - vln) / (sl - sm)
    rho = c * l[0]
    energy = c * (l[1] + l[0] * (sm - vln) * (sm + pl / (l[0] * (sl - vln))))
    star = [sm * l[0] * c, c * l[3]]
    m = [rho * (vl[d] + (star[d] / rho - vln) * n[d]) for d in range(2)]
    tx, ty = x + torch.sign(n[0]).long(), y + torch.sign(n[1]).long()
    inside = (tx >= 0) & (tx < nx) & (ty >= 0) & (ty < ny)
    t, index, value = (ty * nx + tx)[inside], (y * nx + x)[inside], torch.stack([rho, energy] + m)[:, inside]
    last = torch.full((ny * nx,), -1, dtype=torch.int64, device=t.device).scatter_reduce_(0, t, index, "amax")
    win = last[t] == index        # of several sources of one cell, the highest index
    out = ua.reshape(4, -1).clone()
    out[:, t[win]] = value[:, win]
    return out.view(4, ny, nx)


def _extrapolate(u, phi, h):
    band = (phi >= h) & (phi <= 6 * h * math.sqrt(0.5))
    q = _mirror(phi.unsqueeze(0), 0, 1)[0]
    xm, xp, ym, yp = q[1:-1, :-2], q[1:-1, 2:], q[:-2, 1:-1], q[2:, 1:-1]
    gx, gy = xp - xm, yp - ym
    s = torch.sqrt(gx * gx + gy * gy)
    wx, wy = (gx / s).abs(), (gy / s).abs()
    l1 = wx + wy
    use = l1 > 1e-2
    wx, wy = torch.where(use, wx / l1, 0.5), torch.where(use, wy / l1, 0.5)
    for _ in range(64):
        g = _mirror(u, 0, 1)
        px = torch.where(xm < xp, g[:, 1:-1, :-2], g[:, 1:-1, 2:])
        py = torch.where(ym < yp, g[:, :-2, 1:-1], g[:, 2:, 1:-1])
        new = px * wx + py * wy
        new = torch.where(band & ~torch.isnan(new).any(0), new, u)
        moved = (new - u).abs().sum(0).max()
        u = new
        if float(moved) < 1e-8:
            break
    return u

"""Performance cases of culbm_b200: the work its users have it do, through its
public entry points.

* ``host``: one run from an init state in host memory to the four fields in
  host memory (``Simulation.run_host``, page-locked arrays): what
  ``single_dev_expt_main`` does between its init-state folder and its dump.
* ``interval``: a running simulation advanced by one dump interval
  (``step``, ``moments``, ``fields``, ``mass_momentum``): the driver's
  ``--dstep`` loop, and a program that watches a run.
* ``gradient``: J and its gradients from the discrete adjoint
  (``AdjointProblem.gradient``), soft field and inlet set beforehand.
* ``design``: one design-optimisation step through the torch shim
  (``PressureDrop.apply`` and ``backward``).

Scenes are the seeded channels of ``culbm_b200.scenes`` (equilibrium inlet and
outlet on the x faces, bounce-back y and z faces, solid spheres or a soft
obstacle field), built on the GPU, with a few percent of inlet turbulence so
that every velocity component carries a signal.
"""
import math

import numpy as np
import torch

import culbm_b200
from culbm_b200 import adjoint, scenes

HBM = {"fp32": 4, "fp16": 2, "bf16": 2, "fp16sr": 2, "bf16sr": 2, "fp64": 8}   # bytes of a stored population
FLOPS_STEP = 300       # of one cell update (moments, 27 equilibria, relaxation)
FLOPS_ADJOINT = 600    # of one reverse cell update


def _host(name, domain, storage, stream, steps, opt=0, tile=(0, 0, 0), inner=0, kind="host"):
    c = {"kind": kind, "nx": domain[0], "ny": domain[1], "nz": domain[2], "storage": storage, "stream": stream,
         "opt": opt, "tx": tile[0], "ty": tile[1], "tz": tile[2], "inner": inner, "steps": steps}
    return dict(c, name=name) if name else c


def _grad(name, domain, storage, t0, t1, every, checkpoint="", kind="gradient"):
    c = {"kind": kind, "nx": domain[0], "ny": domain[1], "nz": domain[2], "storage": storage, "t0": t0, "t1": t1,
         "every": every, "checkpoint": checkpoint}
    return dict(c, name=name) if name else c


def listed():
    return [
        # A test-sized scene watched every ten steps: launches and host latency.
        _host("interval 32x16x16 inplace", (32, 16, 16), "fp32", 1, 10, kind="interval"),
        # The 64^3 sphere channel, 200 steps of the plain pull: the whole state fits in L2.
        _host("run 64^3 pull", (64, 64, 64), "fp32", 0, 200),
        # The reference's headline domain, in place and with the double buffer.
        _host("run 288 inplace", (288, 272, 280), "fp32", 1, 100),
        _host("run 288 pull", (288, 272, 280), "fp32", 0, 100),
        # 16-bit populations with stochastic rounding: the mixed-precision runs.
        _host("run 288 pull fp16sr", (288, 272, 280), "fp16sr", 0, 100),
        _host("run 512 inplace fp16sr", (512, 512, 256), "fp16sr", 1, 60),
        # A domain cut from a measured geometry: no extent is a multiple of anything.
        _host("run 211x157x149 bf16sr", (211, 157, 149), "bf16sr", 1, 100),
        # The reference's blocked policies: (1,3) with its documented tile on the
        # headline domain, and pull tiles with the driver's default domain and tile.
        _host("blocked 288 inplace", (288, 272, 280), "fp32", 1, 50, 3, (64, 96, 76), 5),
        _host("blocked 256^3 pull", (256, 256, 256), "fp32", 0, 50, 3, (64, 48, 38), 5),
        # The FP64 run that the other formats' errors are stated against.
        _host("run 128x128x64 fp64", (128, 128, 64), "fp64", 0, 200),
        # The 128x64x64 soft-obstacle channel: one step of a design loop in torch.
        _grad("design 128x64x64", (128, 64, 64), "fp32", 300, 500, 50, kind="design"),
        # A larger one with 16-bit states and checkpoints.
        _grad("gradient 192x136x140 fp16sr", (192, 136, 140), "fp16sr", 90, 150, 12),
    ]


def _extent(rng, lo, hi):
    """Log-uniform in [lo, hi]; every other one is a multiple of 8."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v // 8 * 8) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["host", "host", "host", "interval", "blocked", "blocked", "gradient", "design"])
    if kind in ("gradient", "design"):
        while True:
            d = (_extent(rng, 32, 224), _extent(rng, 16, 144), _extent(rng, 16, 144))
            if d[0] * d[1] * d[2] < 2_500_000:
                break
        t1 = rng.randint(40, 200)
        storage = rng.choice(["fp32", "fp32", "fp16sr"])
        mixed = "fp16sr" if storage == "fp32" and rng.random() < 0.3 else ""
        return _grad("", d, storage, rng.randint(t1 // 3, t1 - 1), t1, rng.randint(5, 25), mixed, kind)
    top = 64 if kind == "interval" else 416
    while True:
        d = tuple(_extent(rng, 24, top) for _ in range(3))
        n = d[0] * d[1] * d[2]
        if n < 40_000_000:
            break
    if kind == "blocked":
        storage = rng.choice(["fp32", "fp32", "fp16sr"])
        inner = rng.randint(2, 5)
        tile = (rng.choice([64, 96, 128, 160]), rng.choice([32, 48, 64]), rng.choice([32, 38, 48]))
        steps = min(rng.randint(10, 60), max(10, int(1e9 / n)))
        return _host("", d, storage, rng.randint(0, 1), steps, rng.choice([1, 3, 3]), tile, inner)
    storage = rng.choice(["fp32", "fp32", "fp32", "fp16sr", "fp16sr", "fp16", "bf16sr", "bf16", "fp64"])
    if n > 8_000_000 and storage == "fp64":
        storage = "fp32"
    steps = rng.randint(5, 40)
    if kind == "host":
        steps = min(rng.randint(20, 200), max(10, int(3.5e11 / (n * 54 * HBM[storage]))))
    return _host("", d, storage, rng.randint(0, 1), steps, kind=kind)


# ------------------------------------------------------------------- inputs ---

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _scene(case, seed):
    """flag (int32), rho, vx, vy, vz and the soft field, shape (nz, ny, nx), on the device."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev, rng = _device(), np.random.default_rng(seed)
    soft_model = case["kind"] in ("gradient", "design")
    flag = torch.full((nz, ny, nx), scenes.FLUID, dtype=torch.int32, device=dev)
    z = torch.arange(nz, device=dev).view(-1, 1, 1)
    y = torch.arange(ny, device=dev).view(1, -1, 1)
    x = torch.arange(nx, device=dev).view(1, 1, -1)
    if not soft_model:
        # 40 spheres of radius 4 to 12 on the headline domain; as dense and in proportion elsewhere
        n, short = nx * ny * nz, min(nx, ny, nz)
        for _ in range(max(1, min(120, n // 548_000))):
            r = rng.uniform(4.0, 12.0) if short >= 128 else rng.uniform(0.08, 0.14) * short
            c = [rng.uniform(0.1 * e, 0.9 * e) for e in (nx, ny, nz)]
            box = tuple(slice(max(0, int(q - r)), int(q + r) + 2) for q in c[::-1])
            m = ((z[box[0]] - c[2]) ** 2 + (y[:, box[1]] - c[1]) ** 2 + (x[:, :, box[2]] - c[0]) ** 2) < r * r
            flag[box][m] = scenes.WALL
    flag[:, :, (0, -1)] = scenes.EQUILIBRIUM
    flag[:, (0, -1), :] = scenes.WALL
    flag[(0, -1), :, :] = scenes.WALL
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    noise = torch.rand((3, nz, ny), generator=gen, device=dev) - 0.5
    u_in = 0.02 if (nx, ny, nz) == (64, 64, 64) else 0.05
    if soft_model:   # parabolic profile of peak 0.04
        py = (4.0 * ((y - 0.5) / (ny - 2)) * (1.0 - (y - 0.5) / (ny - 2))).clamp(min=0)
        pz = (4.0 * ((z - 0.5) / (nz - 2)) * (1.0 - (z - 0.5) / (nz - 2))).clamp(min=0)
        u_in = 0.04 * (pz * py)[:, :, 0]
    rho = torch.ones((nz, ny, nx), device=dev)
    u = torch.zeros((3, nz, ny, nx), device=dev)
    inlet = (flag[:, :, 0] == scenes.EQUILIBRIUM)
    u[0, :, :, 0] = torch.where(inlet, u_in * (1.0 + 0.2 * noise[0]), torch.zeros_like(noise[0]))
    u[1, :, :, 0] = torch.where(inlet, u_in * 0.2 * noise[1], torch.zeros_like(noise[1]))
    u[2, :, :, 0] = torch.where(inlet, u_in * 0.2 * noise[2], torch.zeros_like(noise[2]))
    soft = None
    if soft_model:
        soft = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
        for _ in range(16):
            c = [rng.uniform(0.15 * e, 0.85 * e) for e in (nx, ny, nz)]
            s = rng.uniform(3.0, 8.0)
            soft += torch.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2.0 * s * s))
        soft = soft.clamp(0.0, 1.0).float()
        soft[flag != scenes.FLUID] = 0.0
    return flag, rho, u, soft


def _pinned(t, dtype=None):
    """A page-locked host array with the values of tensor t, as numpy."""
    h = torch.empty(t.numel(), dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t.reshape(-1))
    a = h.numpy()
    return a.view(dtype) if dtype else a


def _simulation(case):
    kw = {}
    if case["opt"]:
        kw = {"tile": (case["tx"], case["ty"], case["tz"]), "inner_loop": case["inner"]}
    return culbm_b200.Simulation((case["nx"], case["ny"], case["nz"]), stream_policy=case["stream"],
                                 opt_policy=case["opt"], inv_tau=0.5, storage=case["storage"], **kw)


def _problem(case):
    return adjoint.AdjointProblem((case["nx"], case["ny"], case["nz"]), window=(case["t0"], case["t1"]), inv_tau=0.5,
                                  checkpoint_every=case["every"], storage=case["storage"],
                                  checkpoint_storage=case["checkpoint"] or None)


def prepare(case, seed):
    flag, rho, u, soft = _scene(case, seed)
    arrs = [_pinned(flag, np.uint32)] + [_pinned(t) for t in (rho, u[0], u[1], u[2])]
    state = {"case": case, "in": arrs}
    if case["kind"] == "host":
        state["sim"] = _simulation(case)
        state["out"] = tuple(_pinned(torch.zeros_like(rho)) for _ in range(4))
    elif case["kind"] == "interval":
        state["sim"] = _simulation(case)
        state["sim"].load_state(*arrs)
    elif case["kind"] == "gradient":
        state["problem"] = _problem(case)
        state["problem"].set_state(*arrs, soft=_pinned(soft))
    else:
        state["problem"] = _problem(case)
        state["drop"] = adjoint.PressureDrop(state["problem"], arrs[0], arrs[1], arrs[3], arrs[4])
        state["soft"] = soft.reshape(-1)
        state["inv_tau"] = torch.tensor(0.5, device=soft.device)
        state["inlet"] = u[0].reshape(-1).clone()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "host":
        return state["sim"].run_host(case["steps"], *state["in"], out=state["out"])
    if case["kind"] == "interval":
        sim = state["sim"]
        sim.step(case["steps"])
        sim.moments()
        return sim.fields(), sim.mass_momentum()
    if case["kind"] == "gradient":
        return state["problem"].gradient()
    params = [t.detach().requires_grad_() for t in (state["soft"], state["inv_tau"], state["inlet"])]
    J = state["drop"].apply(*params)
    J.backward()
    return J.detach(), params[0].grad, params[1].grad, params[2].grad


def work(case):
    """Populations read and written once per step (and the adjoint's), op bytes, and the arrays in and out."""
    n, s = case["nx"] * case["ny"] * case["nz"], HBM[case["storage"]]
    if case["kind"] in ("host", "interval"):
        per_step = n * (54 * s + 1)
        io = n * 16 + (n * 20 if case["kind"] == "host" else n * 27 * s)
        return {"bytes": float(case["steps"] * per_step + io), "flops": float(FLOPS_STEP * n * case["steps"])}
    t = case["t1"]
    c = HBM[case["checkpoint"]] if case["checkpoint"] else s
    forward = n * (54 * s + 5)               # state in and out, op byte, soft value
    again = n * (54 * c + 5)                 # recomputation between checkpoints
    back = n * (27 * c + 54 * 4 + 16 + 5)    # state in, adjoint populations in and out, dJ/ds read and written
    return {"bytes": float(t * (forward + again + back)),
            "flops": float(n * t * (2 * FLOPS_STEP + FLOPS_ADJOINT))}


def tolerance(case):
    """About four times the measured distance from the 64-bit run: FP32 sums in
    another order, or other rounding of the 16-bit populations."""
    if case["storage"] == "fp64":
        return {"rel": 1.5e-7}   # the fields leave as FP32
    if case["kind"] in ("host", "interval"):
        return {"rel": {"fp32": 5e-5, "fp16": 1.2e-2, "fp16sr": 1.2e-2, "bf16": 3e-2, "bf16sr": 3e-2}[case["storage"]]}
    return {"rel": 3e-5 if case["storage"] == "fp32" and not case["checkpoint"] else 1e-4}


# ---------------------------------------------------------- 64-bit reference ---

_C = [(d % 3 - 1, d // 3 % 3 - 1, d // 9 - 1) for d in range(27)]
_W = [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[sum(map(abs, c))] for c in _C]


def _shift(t, k, dim):
    """Values pulled from one cell back along `dim` (k = +-1), a cell at the face from itself."""
    n = t.shape[dim]
    if k == 0 or n == 1:
        return t
    if k > 0:
        return torch.cat([t.narrow(dim, 0, 1), t.narrow(dim, 0, n - 1)], dim)
    return torch.cat([t.narrow(dim, 1, n - 1), t.narrow(dim, n - 1, 1)], dim)


def _pulled(f):
    return torch.stack([_shift(_shift(_shift(f[d], cx, 2), cy, 1), cz, 0) for d, (cx, cy, cz) in enumerate(_C)])


def _moments(g):
    rho = 1.0 + g.sum(0)
    j = [sum((c[q] * g[d] for d, c in enumerate(_C) if c[q]), torch.zeros_like(rho)) for q in range(3)]
    return rho, [v / rho for v in j]


def _equilibrium(rho, u):
    uu = 1.0 - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    out = []
    for (cx, cy, cz), w in zip(_C, _W):
        cu = 3.0 * (cx * u[0] + cy * u[1] + cz * u[2])
        out.append(w * (rho * (uu + cu + 0.5 * cu * cu) - 1.0))
    return torch.stack(out)


def _update(g, m, rho, u, omega, soft=None):
    """Post-collision populations of pulled populations g: equilibrium cells, bounce-back, BGK."""
    g = torch.where(m["load"], g, torch.zeros_like(g))
    g = torch.where(m["equ"], _equilibrium(rho, u), g)
    b = g.flip(0)
    g, b = torch.where(m["bb"], b, g), torch.where(m["bb"], g, b)
    r, v = _moments(g)
    c = omega * _equilibrium(r, v) + (1.0 - omega) * g
    if soft is not None:
        c = c + soft * (b - c)
    return torch.where(m["collide"], c, g)


def _masks(flag):
    return {k: (flag & b) != 0 for k, b in (("load", scenes.LOAD), ("equ", scenes.EQU), ("bb", scenes.BOUNCE_BACK),
                                            ("collide", scenes.COLLIDE), ("dump", scenes.DUMP_RHO))}


def _exact_run(case, seed):
    flag, rho, u, _ = _scene(case, seed)
    m, rho, u = _masks(flag), rho.double(), [v.double() for v in u]
    f = torch.zeros((27,) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
    for _ in range(case["steps"]):
        f = _update(_pulled(f), m, rho, u, 0.5)
    g = _pulled(f)
    r, v = _moments(g)
    out = [torch.where(m["dump"], a, b).reshape(-1) for a, b in zip([r] + v, [rho] + u)]
    if case["kind"] == "host":
        return out
    on = m["load"] | m["equ"]
    j = [sum((c[q] * g[d] for d, c in enumerate(_C) if c[q]), torch.zeros_like(r)) for q in range(3)]
    return out, torch.stack([torch.where(on, t, torch.zeros_like(t)).sum() for t in [r] + j])


def _exact_gradient(case, seed):
    flag, rho, u, soft = _scene(case, seed)
    m = _masks(flag)
    soft = soft.double().requires_grad_()
    mac = [t.double().requires_grad_() for t in (rho, u[0], u[1], u[2])]
    omega = torch.tensor(0.5, dtype=torch.float64, device=rho.device, requires_grad=True)
    params = [soft, omega] + mac
    t0, t1 = case["t0"], case["t1"]
    fluid = m["collide"]
    planes = (1, case["nx"] - 2)
    count = [float(fluid[:, :, p].sum()) for p in planes]

    def objective(g):
        r = (1.0 + g.sum(0)) / 3.0
        a, b = ((torch.where(fluid[:, :, p], r[:, :, p], torch.zeros_like(r[:, :, p]))).sum() / c
                for p, c in zip(planes, count))
        return (a - b) / (t1 - t0 + 1)

    def step(f):
        return _update(_pulled(f), m, mac[0], mac[1:], omega, soft)

    f = torch.zeros((27,) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
    keep, J, K = {0: f}, 0.0, max(1, int(math.sqrt(t1)))
    with torch.no_grad():
        for t in range(t1 + 1):
            if t >= t0:
                J += float(objective(_pulled(f)))
            if t % K == 0:
                keep[t] = f
            if t < t1:
                f = step(f)
    grads = [torch.zeros_like(p) for p in params]
    nu = torch.zeros_like(f)

    def back(f, t, nu):
        f = f.detach().requires_grad_()
        total = torch.zeros((), dtype=torch.float64, device=f.device)
        if t < t1:
            total = total + (step(f) * nu).sum()
        if t >= t0:
            total = total + objective(_pulled(f))
        got = torch.autograd.grad(total, [f] + params, allow_unused=True)
        for a, b in zip(grads, got[1:]):
            if b is not None:
                a += b
        return got[0]

    t = t1
    while t >= 0:
        first = t // K * K
        states = [keep.pop(first)]
        with torch.no_grad():
            for _ in range(first, t):
                states.append(step(states[-1]))
        while t >= first:
            if t < t1 or t >= t0:
                nu = back(states.pop(), t, nu)
            t -= 1
    gs = torch.where(fluid, grads[0], torch.zeros_like(grads[0])).reshape(-1)
    gm = torch.stack([torch.where(m["equ"], a, torch.zeros_like(a)).reshape(-1) for a in grads[2:]])
    if case["kind"] == "gradient":
        return J, float(grads[1]), gs, gm
    return torch.tensor(J, dtype=torch.float64), gs, grads[1].detach(), gm[1]


def exact(case, seed):
    if case["kind"] in ("host", "interval"):
        if not torch.cuda.is_available() and case["nx"] * case["ny"] * case["nz"] * case["steps"] > 5e7:
            return None
        return _exact_run(case, seed)
    if not torch.cuda.is_available() and case["nx"] * case["ny"] * case["nz"] * case["t1"] > 5e6:
        return None
    return _exact_gradient(case, seed)

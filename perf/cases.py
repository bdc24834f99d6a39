"""The workloads this library is timed on: solves, batches, coupling steps and
the warm-start network, each through the public entry points (the qesb package
over the C ABI).

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  a user's state before the call: inputs on the GPU, handles, buffers
    run(state)           one pass, and its outputs
    work(case)           bytes and operations the pass cannot do without
    exact(case, seed)    the outputs in 64 bits, by plain torch

The domains are synthetic cities: cuboid buildings placed at random on flat
ground, stair-step wall coefficients, a power-law inflow from a random
direction, built here with torch alone.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qes-public_b200"))

import qesb  # noqa: E402
from qesb import warmstart as ws  # noqa: E402

DEV = "cuda:0"
OMEGA = float(np.float32(1.78))
TOL = 1e-9              # the reference's tolerance: never met in FP32, so a plain solve runs its itermax
ITERMAX = 10000
WINDOW, WINDOW_TOL = 32, 4e-3   # the window stopping rule of the benchmark
PRE_TOL = 2e-3                  # the over-relaxed pre-phase's end
CHANNELS = (16, 32, 64, 128)    # the shipped warm-start network's levels


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a small domain solved for a fixed count: launches and latency are all there is
        dict(name="small_plain", kind="plain", nx=47, ny=41, nz=20, dx=2.0, ratio=1.0, nb=3, iters=100),
        # the reference's drop-in call on host arrays (solve(WGD, itermax)): the 100 x 100 x 50 cuboid domain
        dict(name="cuboid100_host", kind="host", nx=100, ny=100, nz=50, dx=1.0, ratio=1.0, nb=1, iters=500),
        # a fire code's coupling loop: new winds each step, every solve from the last lambda
        dict(name="fire_steps", kind="fire", nx=160, ny=144, nz=40, dx=2.0, ratio=1.03, nb=18, steps=4),
        # one evaluation city from lambda = 0 to the stopping rule, with the pre-phase
        dict(name="city256", kind="rule", nx=256, ny=256, nz=64, dx=2.0, ratio=1.03, nb=60),
        # the headline: eight cities, learned start, pre-phase and rule, solved together
        dict(name="city256_batch8", kind="batch", nx=256, ny=256, nz=64, dx=2.0, ratio=1.03, nb=60, count=8,
             uneven=False, learned=True),
        # an ensemble list: cities of uneven, odd sizes solved together
        dict(name="uneven_batch12", kind="batch", nx=256, ny=256, nz=96, dx=2.0, ratio=1.03, nb=24, count=12,
             uneven=True, learned=False),
        # the larger grids, a fixed number of the reference's iterations
        dict(name="city400_plain", kind="plain", nx=400, ny=400, nz=100, dx=2.0, ratio=1.03, nb=60, iters=200),
        dict(name="city800_plain", kind="plain", nx=800, ny=800, nz=128, dx=2.0, ratio=1.03, nb=150, iters=100),
        # cut-cell style coefficients (any value per face): the full-coefficient path, odd sizes
        dict(name="cut_cells", kind="full", nx=151, ny=133, nz=61, dx=2.0, ratio=1.03, nb=20, iters=200),
        # the solve for callers that own all device memory
        dict(name="noalloc", kind="noalloc", nx=128, ny=128, nz=48, dx=2.0, ratio=1.03, nb=16, iters=200),
        # the warm-start network alone: inference on the half-resolution grid of a 256 x 256 x 64 domain
        dict(name="net_forward", kind="forward", d=32, h=128, w=128),
        # one training step of it on the half-resolution grid of a 128 x 128 x 64 domain
        dict(name="net_train", kind="train", d=32, h=64, w=64),
    ]


def draw(rng: random.Random):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["plain", "plain", "host", "fire", "rule", "rule", "batch", "batch", "full", "noalloc", "forward",
                       "train"])
    if kind in ("forward", "train"):  # every size a multiple of 8 (four levels)
        big = kind == "forward"
        return dict(kind=kind, d=8 * rng.randint(1, 4), h=8 * rng.randint(3, 16 if big else 8),
                    w=rng.choice([32, 64, 128] if big else [32, 64]) if rng.random() < 0.7
                    else 8 * rng.randint(3, 16 if big else 8))
    c = dict(kind=kind, dx=rng.choice([1.0, 2.0]), ratio=rng.choice([1.0, 1.02, 1.03]))
    if kind == "plain":
        c.update(nx=logint(32, 600), ny=logint(32, 600), nz=logint(16, 110), iters=logint(50, 200))
    elif kind == "host":
        c.update(nx=logint(32, 200), ny=logint(32, 200), nz=logint(16, 64), iters=logint(100, 500))
    elif kind == "fire":
        c.update(nx=logint(64, 200), ny=logint(64, 200), nz=logint(24, 64), steps=rng.randint(2, 4))
    elif kind == "rule":
        c.update(nx=logint(64, 320), ny=logint(64, 320), nz=logint(32, 96))
    elif kind == "batch":
        learned = rng.random() < 0.4
        if learned:  # the network's grid: multiples of 16
            c.update(nx=16 * rng.randint(4, 16), ny=16 * rng.randint(4, 16), nz=16 * rng.randint(2, 4))
        else:
            c.update(nx=logint(64, 256), ny=logint(64, 256), nz=logint(32, 96))
        c.update(count=rng.randint(2, 8), uneven=not learned and rng.random() < 0.6, learned=learned)
    else:
        c.update(nx=logint(32, 200), ny=logint(32, 200), nz=logint(16, 64), iters=logint(50, 200))
    # buildings as dense as the 400 x 400 city's
    c["nb"] = max(1, int(round(60 * c["nx"] * c["ny"] / 160000)))
    return c


# ---------------------------------------------------------------------------
# synthetic domains (torch, seeded)
# ---------------------------------------------------------------------------
def stretched(nz, ratio):
    """dz_array: 1 m at the ground, stretched by `ratio`; index 0 is the ghost layer."""
    dz = np.empty(nz + 1, np.float32)
    dz[1:] = ratio ** np.arange(nz)
    dz[0] = dz[1]
    return dz


def city(nx, ny, nz, dx, ratio, nb, seed, cut=False):
    """Flags, coefficients and initial winds as device tensors in the
    reference's layouts ((z, y, x) views), and dz (numpy, with the ghost layer)."""
    r = random.Random(seed)
    dz = stretched(nz, ratio)
    top = np.concatenate([[0.0], np.cumsum(dz[1:].astype(np.float64))])  # upper face of layer k at top[k]
    zc = np.concatenate([[-0.5 * dz[0]], 0.5 * (top[1:] + top[:-1])])
    Z, Y, X = nz + 1, ny, nx
    flag = torch.ones(Z, Y, X, dtype=torch.int32, device=DEV)
    flag[0] = 2
    for _ in range(nb):  # footprints 10-40 m, heights 10-60 m, two cells clear of the sides
        lx = min(max(2, int(r.uniform(10, 40) / dx)), max(2, X // 3))
        ly = min(max(2, int(r.uniform(10, 40) / dx)), max(2, Y // 3))
        hz = int(np.searchsorted(zc, r.uniform(10, 60)))
        hz = min(max(hz, 2), max(2, (2 * nz) // 3))
        i, j = r.randint(2, X - 3 - lx), r.randint(2, Y - 3 - ly)
        flag[1:hz, j:j + ly, i:i + lx] = 0
    solid = flag != 1
    d = torch.from_numpy(dz).to(DEV)
    co = {q: torch.ones(Z, Y, X, device=DEV) for q in "efghmn"}
    k = slice(1, Z - 1)
    fluid = ~solid[k]
    open_ = {q: torch.ones_like(fluid) for q in "efghmn"}
    open_["e"][:, :, :-1] = ~solid[k, :, 1:]
    open_["f"][:, :, 1:] = ~solid[k, :, :-1]
    open_["g"][:, :-1] = ~solid[k, 1:]
    open_["h"][:, 1:] = ~solid[k, :-1]
    open_["m"] = ~solid[2:]
    open_["n"] = ~solid[:Z - 2]
    dm = (d[1:Z - 1] * 0.5 * (d[1:Z - 1] + d[2:])).view(-1, 1, 1)
    dn = (d[1:Z - 1] * 0.5 * (d[1:Z - 1] + d[:Z - 2])).view(-1, 1, 1)
    div = dict(e=dx * dx, f=dx * dx, g=dx * dx, h=dx * dx, m=dm, n=dn)
    for q in "efghmn":
        co[q][k] = (open_[q] | ~fluid).float() / div[q]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    if cut:  # partly covered faces beside the walls and in one cell of twenty elsewhere
        near = ~(open_["e"] & open_["f"] & open_["g"] & open_["h"] & open_["m"]) | (
            torch.rand(fluid.shape, generator=gen, device=DEV) < 0.05)
        for q in "efghmn":
            frac = 0.05 + 0.95 * torch.rand(fluid.shape, generator=gen, device=DEV)
            co[q][k] = torch.where(near & fluid, co[q][k] * frac, co[q][k])
    uref, p, th = r.uniform(3, 10), r.uniform(0.1, 0.3), r.uniform(0, 2 * math.pi)
    prof = np.zeros(Z + 1)
    prof[1:Z] = uref * (np.maximum(zc[1:], 0.1) / 10.0) ** p
    prof = torch.from_numpy(prof.astype(np.float32)).to(DEV).view(-1, 1, 1)
    u0 = (math.cos(th) * prof).expand(Z + 1, Y + 1, X + 1).contiguous()
    v0 = (math.sin(th) * prof).expand(Z + 1, Y + 1, X + 1).contiguous()
    w0 = torch.zeros(Z + 1, Y + 1, X + 1, device=DEV)
    c = dict(flag=flag, u0=u0, v0=v0, w0=w0, **co)
    zero_solid_faces(c["u0"], c["v0"], c["w0"], solid)
    return c, dz


def zero_solid_faces(u, v, w, solid):
    """The faces of solid cells carry no flow (the ground's top face included)."""
    Z, Y, X = solid.shape
    for t, (a, b, c) in ((u, (0, 0, 1)), (v, (0, 1, 0)), (w, (1, 0, 0))):
        t[:Z, :Y, :X].masked_fill_(solid, 0.0)
        t[a:Z + a, b:Y + b, c:X + c].masked_fill_(solid, 0.0)


def fire_winds(c, dx, t):
    """A fire's winds added to a city's: a Gaussian updraft and a convergent
    inflow around a centre that moves with the step t."""
    Zf, Yf, Xf = c["u0"].shape
    y = torch.arange(Yf, device=DEV, dtype=torch.float32).view(1, -1, 1) * dx
    x = torch.arange(Xf, device=DEV, dtype=torch.float32).view(1, 1, -1) * dx
    cx, cy = 0.3 * Xf * dx + 4.0 * t, 0.5 * Yf * dx
    g = torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * 20.0 ** 2))
    k = torch.arange(Zf, device=DEV, dtype=torch.float32).view(-1, 1, 1) / Zf
    out = dict(c)
    out["u0"] = c["u0"] - (1 - k) * g * (x - cx) / 20.0
    out["v0"] = c["v0"] - (1 - k) * g * (y - cy) / 20.0
    out["w0"] = c["w0"] + 3.0 * g * k * (1 - k)
    zero_solid_faces(out["u0"], out["v0"], out["w0"], c["flag"] != 1)
    return out


def sizes(case, i):
    """Grid of domain i of a case (an uneven batch's domains shrink by odd steps)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if not case.get("uneven"):
        return nx, ny, nz
    r = random.Random(1000 * nx + 10 * ny + nz + 7919 * i)
    pick = lambda a, b: b if a >= b else r.randint(a, b)  # noqa: E731
    return pick(64, nx), pick(64, ny), pick(32, nz)


def domains(case, seed):
    """[(arrays, dz, (nx, ny, nz))] of a case."""
    out = []
    for i in range(case.get("count", 1)):
        nx, ny, nz = sizes(case, i)
        nb = case["nb"] if not case.get("uneven") else max(1, int(round(60 * nx * ny / 160000)))
        c, dz = city(nx, ny, nz, case["dx"], case["ratio"], nb, 7919 * seed + i,
                     cut=case["kind"] in ("full", "noalloc"))
        out.append((c, dz, (nx, ny, nz)))
    return out


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
INPUTS = ("e", "f", "g", "h", "m", "n", "flag", "u0", "v0", "w0")


def domain_of(case, dz, n):
    return qesb.Domain(n[0], n[1], n[2], case["dx"], case["dx"], float(dz.min()), dz)


def solver_for(case, dz, n):
    return qesb.SolverFactory.create(qesb.B200_Type, domain_of(case, dz, n), TOL)


def give(s, c):
    s.set_inputs_device(*[c[q].data_ptr() for q in INPUTS])


def to_rule(s, n):
    """The pre-phase and stopping rule a production solve runs with."""
    s.set_window_rule(WINDOW, WINDOW_TOL)
    s.set_prephase(qesb.prephase_omega(n[0], n[1]), PRE_TOL, ITERMAX)


def wind_buffers(c):
    return [torch.empty_like(c["u0"]) for _ in range(3)]


def net_weights(seed):
    """FP32 weights and biases of the network: He-scaled, the head's small."""
    g = torch.Generator().manual_seed(seed)
    L = len(CHANNELS)
    out = {}

    def layer(name, cin, cout, used_in=None, used_out=None, std=None):
        w = torch.randn(27, cin, cout, generator=g) * (std or math.sqrt(2.0 / (27 * (used_in or cin))))
        b = torch.randn(cout, generator=g) * 0.05
        if used_in:
            w[:, used_in:] = 0.0
        if used_out:
            w[:, :, used_out:] = 0.0
            b[used_out:] = 0.0
        out[name] = (w, b)

    for l in range(L):
        layer(f"e{l}a", 16 if l == 0 else CHANNELS[l - 1], CHANNELS[l], used_in=5 if l == 0 else None)
        layer(f"e{l}", CHANNELS[l], CHANNELS[l])
    for l in range(L - 2, -1, -1):
        layer(f"d{l}a", CHANNELS[l + 1] + CHANNELS[l], CHANNELS[l])
        layer(f"d{l}", CHANNELS[l], CHANNELS[l])
    layer("head", CHANNELS[0], 16, used_out=1, std=0.05)
    return out


def net_input(case, seed):
    """Network input (z, y, x, 16) BF16, target and weight (z, y, x) FP32, as
    a domain gives them: a sparse scaled divergence, flags, smooth profiles."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    D, H, W = case["d"], case["h"], case["w"]
    x = torch.zeros(D, H, W, 16, device=DEV)
    near = torch.rand(D, H, W, generator=g, device=DEV) < 0.1
    x[..., 0] = torch.randn(D, H, W, generator=g, device=DEV) * near * 0.3
    x[..., 1] = (torch.rand(D, H, W, generator=g, device=DEV) < 0.05).float()
    x[..., 2] = (0.5 + torch.linspace(0, 1, D, device=DEV)).view(-1, 1, 1)
    x[:, 0, :, 3] = x[:, -1, :, 3] = x[:, :, 0, 3] = x[:, :, -1, 3] = 1.0
    x[..., 4] = torch.linspace(0, 1, D, device=DEV).view(-1, 1, 1)
    tgt = torch.randn(D, H, W, generator=g, device=DEV)
    wgt = (x[..., 3] == 0).float()
    return x.to(torch.bfloat16), tgt, wgt


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        net = ws.WarmStartNet(device=0, channels=CHANNELS)
        for name, (w, b) in net_weights(seed).items():
            net.layers[name].W.copy_(w.reshape(-1))
            net.layers[name].b.copy_(b)
        torch.cuda.synchronize()
        for layer in net.layers.values():
            layer.sync()
        s = ws.Shapes(case["d"], case["h"], case["w"])
        x, tgt, wgt = net_input(case, seed)
        net._bufs(s)["x"].copy_(x.reshape(-1))
        return dict(kind=kind, net=net, shape=s, tgt=tgt, wgt=wgt, inv=1.0 / float(wgt.sum()))
    doms = domains(case, seed)
    torch.cuda.synchronize()
    c, dz, n = doms[0]
    if kind == "host":  # the reference's objects, on host arrays
        d = domain_of(case, dz, n)
        wgd = qesb.WINDSGeneralData(d)
        wgd.icellflag = c["flag"].reshape(-1).cpu().numpy()
        for q in INPUTS:
            if q != "flag":
                setattr(wgd, q, c[q].reshape(-1).cpu().numpy())
        return dict(kind=kind, solver=qesb.SolverFactory.create(qesb.B200_Type, d, TOL), wgd=wgd, iters=case["iters"])
    if kind == "noalloc":
        return dict(kind=kind, c=c, domain=domain_of(case, dz, n), out=wind_buffers(c),
                    lam=torch.zeros_like(c["e"]), iters=case["iters"])
    if kind == "batch":
        solvers = [solver_for(case, z, m) for _, z, m in doms]
        for s, (a, _, m) in zip(solvers, doms):
            give(s, a)
            to_rule(s, m)
        net = None
        if case["learned"]:  # the start stage goes with the learned start
            net = ws.WarmNet(device=0)
            for s in solvers:
                s.set_prephase_start(1.8, 8)
        outs = [wind_buffers(a) for a, _, _ in doms]
        qesb.autotune_batch(solvers)  # once per list shape, as the benchmark does
        return dict(kind=kind, solvers=solvers, net=net, doms=doms, out=outs,
                    ptrs=[[o[q].data_ptr() for o in outs] for q in range(3)])
    s = solver_for(case, dz, n)
    if kind in ("rule", "fire"):
        to_rule(s, n)
    if kind in ("rule", "plain"):
        s.set_option("autotune", 1)
    st = dict(kind=kind, solver=s, c=c, out=wind_buffers(c), iters=case.get("iters", ITERMAX))
    if kind == "fire":
        st["steps"] = [fire_winds(c, case["dx"], t) for t in range(case["steps"])]
        torch.cuda.synchronize()
    else:
        give(s, c)
    return st


def run(state):
    kind = state["kind"]
    if kind == "forward":
        return state["net"].forward(state["shape"])
    if kind == "train":
        net = state["net"]
        y = net.forward(state["shape"])
        net.backward(state["shape"], state["tgt"], state["wgt"], state["inv"])
        net.adam(1e-5)
        return dict(y=y, loss=net.loss, grads={k: [L.dW, L.db] for k, L in net.layers.items()})
    if kind == "host":
        s, w = state["solver"], state["wgd"]
        s.resetLambda()
        st = s.solve(w, state["iters"])
        return dict(winds=[w.u, w.v, w.w], iterations=st["iterations"])
    if kind == "noalloc":
        state["lam"].zero_()
        torch.cuda.current_stream().synchronize()
        c = state["c"]
        st = qesb.solve_noalloc(state["domain"], TOL, state["iters"], *[c[q].data_ptr() for q in INPUTS],
                                state["lam"].data_ptr(), *[o.data_ptr() for o in state["out"]])
        return dict(winds=state["out"], lam=state["lam"], iterations=st["iterations"])
    if kind == "batch":
        solvers = state["solvers"]
        if state["net"] is not None:
            state["net"].warm_start_batch(solvers)
        else:
            for s in solvers:
                s.resetLambda()
        st = qesb.solve_batch(solvers, ITERMAX, *state["ptrs"])
        return dict(winds=state["out"], iterations=[[x["pre_iterations"], x["iterations"]] for x in st])
    s = state["solver"]
    s.resetLambda()
    ptrs = [o.data_ptr() for o in state["out"]]
    its = []
    for c in state.get("steps", (None,)):
        if c is not None:
            give(s, c)
        st = s.solve_device(state["iters"], *ptrs)
        its.append([st["pre_iterations"], st["iterations"]])
    return dict(winds=state["out"], iterations=its)


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        V = case["d"] * case["h"] * case["w"]
        fl = by = 0
        for name, (w, b) in net_weights(0).items():
            v = V >> (3 * (0 if name == "head" else int(name[1])))
            first = kind == "train" and name == "e0a"  # no input gradient
            fl += 2 * w.numel() * v * (1 if kind == "forward" else 2 if first else 3)
            by += 4 * w.numel() * (1 if kind == "forward" else 8)  # and the gradient, moments and updates
        return dict(bytes=by + V * (2 * 16 + 4 * 16 + (8 if kind == "train" else 0)), flops=fl)
    fl = by = 0
    for i in range(case.get("count", 1)):
        nx, ny, nz = sizes(case, i)
        cells, faces = nx * ny * (nz + 1), (nx + 1) * (ny + 1) * (nz + 2)
        steps = case.get("steps", 1)
        # to the rule: about this many sweeps (pre-phase and reference loop) at this size
        n = case["iters"] if "iters" in case else 1.4 * max(nx, ny) + 64
        fl += steps * n * cells * 17
        by += steps * (7 * 4 * cells + 6 * 4 * faces)  # coefficients and flags, winds in and out
    return dict(bytes=by, flops=fl)


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
class Sor64:
    """Red-black SOR of one domain in FP64 (torch): the reference's equations."""

    def __init__(self, c, dz, dx):
        Z, Y, X = c["flag"].shape
        self.c, self.dx = c, dx
        self.dz = torch.from_numpy(dz).to(DEV).double().view(-1, 1, 1)
        k, j, i = (slice(1, n - 1) for n in (Z, Y, X))
        self.inner = (k, j, i)
        d = self.dz
        u0, v0, w0 = (c[q].double() for q in ("u0", "v0", "w0"))
        co = {q: c[q][k, j, i].double() for q in "efghmn"}
        div = (co["e"] * u0[k, j, 2:X] - co["f"] * u0[k, j, i]) * dx
        div += (co["g"] * v0[k, 2:Y, i] - co["h"] * v0[k, j, i]) * dx
        div += co["m"] * d[k] * 0.5 * (d[k] + d[2:]) * w0[2:Z, j, i]
        div -= co["n"] * d[k] * 0.5 * (d[k] + d[:Z - 2]) * w0[k, j, i]
        self.R = div.mul_(-2.0)
        self.co = co
        self.inv = 1.0 / (co["e"] + co["f"] + co["g"] + co["h"] + co["m"] + co["n"])
        par = (torch.arange(Z, device=DEV).view(-1, 1, 1) + torch.arange(Y, device=DEV).view(1, -1, 1) +
               torch.arange(X, device=DEV).view(1, 1, -1)) % 2
        self.colour = [(par == q)[k, j, i] for q in (0, 1)]
        self.L = torch.zeros(Z, Y, X, dtype=torch.float64, device=DEV)

    def sweeps(self, n, omega):
        L, co, (k, j, i) = self.L, self.co, self.inner
        Z, Y, X = L.shape
        scale = omega * self.inv
        acc = torch.empty_like(self.R)
        for _ in range(n):
            for q in (0, 1):
                torch.mul(co["e"], L[k, j, 2:], out=acc)
                acc.addcmul_(co["f"], L[k, j, :X - 2])
                acc.addcmul_(co["g"], L[k, 2:, i])
                acc.addcmul_(co["h"], L[k, :Y - 2, i])
                acc.addcmul_(co["m"], L[2:, j, i])
                acc.addcmul_(co["n"], L[:Z - 2, j, i])
                acc.sub_(self.R).mul_(scale).add_(L[k, j, i], alpha=1.0 - omega)
                L[k, j, i] = torch.where(self.colour[q], acc, L[k, j, i])
            L[0] = L[1]

    def winds(self):
        c, L, dx = self.c, self.L, self.dx
        Z, Y, X = L.shape
        u, v, w = (c[q].double() for q in ("u0", "v0", "w0"))
        k, j, i = slice(1, Z - 1), slice(1, Y), slice(1, X)
        u[k, j, i] += 0.5 * dx * c["f"][k, j, i].double() * (L[k, j, i] - L[k, j, :X - 1])
        v[k, j, i] += 0.5 * dx * c["h"][k, j, i].double() * (L[k, j, i] - L[k, :Y - 1, i])
        w[k, j, i] += 0.5 * self.dz[k] * c["n"][k, j, i].double() * (L[k, j, i] - L[:Z - 2, j, i])
        solid = c["flag"] != 1
        solid[0] = False  # the solver zeroes the faces of solid cells above the ground layer
        zero_solid_faces(u, v, w, solid)
        return [u, v, w]


def exact_network(case, seed):
    import torch.nn.functional as F

    x, tgt, wgt = net_input(case, seed)
    train = case["kind"] == "train"
    par = {}
    for name, (w, b) in net_weights(seed).items():
        t = w.double().to(DEV).permute(2, 1, 0).reshape(w.shape[2], w.shape[1], 3, 3, 3).contiguous()
        par[name] = (t.requires_grad_(train), b.double().to(DEV).requires_grad_(train))

    def conv(name, t, relu=True):
        y = F.conv3d(t, *par[name], padding=1)
        return torch.relu(y) if relu else y

    L, e, t = len(CHANNELS), [], x.double().permute(3, 0, 1, 2).unsqueeze(0)
    for l in range(L):
        t = F.avg_pool3d(e[-1], 2) if l else t
        e.append(conv(f"e{l}", conv(f"e{l}a", t)))
    d = e[-1]
    for l in range(L - 2, -1, -1):
        d = F.interpolate(d, scale_factor=2, mode="nearest")
        d = conv(f"d{l}", conv(f"d{l}a", torch.cat([d, e[l]], 1)))
    y = conv("head", d, relu=False)
    yv = y[0].permute(1, 2, 3, 0).reshape(-1).detach()
    if not train:
        return yv
    loss = (((y[0, 0] - tgt.double()) * wgt) ** 2).sum() / float(wgt.sum())
    loss.backward()
    grads = {}
    for name, (w, b) in par.items():
        g = w.grad.permute(2, 3, 4, 1, 0).reshape(27 * w.shape[1], w.shape[0])
        gb = b.grad.clone()
        if name == "head":  # channel 0 is the prediction, the others are never trained
            g[:, 1:] = 0.0
            gb[1:] = 0.0
        grads[name] = [g.reshape(-1), gb]
    return dict(y=yv, loss=loss.detach().reshape(1), grads=grads)


def exact(case, seed):
    kind = case["kind"]
    with torch.backends.cudnn.flags(enabled=False):
        if kind in ("forward", "train"):
            return exact_network(case, seed)
    if kind == "fire":  # the converged winds of the last step
        c, dz, n = domains(case, seed)[0]
        doms = [(fire_winds(c, case["dx"], case["steps"] - 1), dz, n)]
    else:
        doms = domains(case, seed)
    res = []
    for c, dz, n in doms:
        if len(res) >= 2:  # two domains of a batch say enough
            res.append([None] * 3)
            continue
        s = Sor64(c, dz, case["dx"])
        if "iters" in case:
            s.sweeps(case["iters"], OMEGA)
        else:  # converged: well past the rule's stop
            m = max(n)
            s.sweeps(5 * m, qesb_free_omega(n))
            s.sweeps(100, 1.5)
        res.append(s.winds())
        if kind == "noalloc":
            return dict(winds=res[0], lam=s.L, iterations=None)
    if kind == "batch":
        return dict(winds=res, iterations=None)
    if kind == "host":
        return dict(winds=[t.reshape(-1).cpu().numpy() for t in res[0]], iterations=None)
    return dict(winds=res[0], iterations=None)


def qesb_free_omega(n):
    return min(1.97, max(1.85, 2.0 - 7.5 / max(n[0], n[1])))

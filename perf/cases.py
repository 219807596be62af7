"""The work that users of this library have it do, as cases that can be timed
and compared: pressure solves through MGSolver, whole time steps through
Simulation, and the U-Net of the learned initial guess through UNet.

A case is a dict of plain values; its "kind" is one of

- "solve":  a variable-density pressure projection from a zero start: the
  density of eight seeded circles and a seeded right-hand side, set_density
  and solve, as a program does for each new density. "sys" mac or fem, m x n
  cells, "box" square ([-1,1]^2, walls all round, the simple spin's) or
  channel (the flag's: [-1,5]x[-1,1], y-periodic, zero pressure at the right
  edge), "mixed" FP32 V-cycles in FP64 defect correction, "krylov" flexible
  conjugate gradients around the V-cycle, "host" NumPy arrays in and out
  instead of device pointers.
- "steps":  "steps" time steps of a simulation and the fields a program
  writes out or checkpoints afterwards. "scene" spin (the rotor in a box),
  sediment (seeded circles and ellipses settling) or flag (the flag in its
  channel); "mixed" as above, "guess" the projections' warm start.
- "infer":  one forward pass of the U-Net on a batch of H x W images.
- "train":  one Adam step of it, and its parameters.
"""
import math

import numpy as np
import torch

from incrmt_b200 import capi, workloads

SQUARE = (-1.0, 1.0, -1.0, 1.0)
CHANNEL = (-1.0, 5.0, -1.0, 1.0)
SEDIMENT = (-0.75, 0.75, -1.5, 1.5)


def listed():
    return [
        # A small projection handed over in host arrays, as a CPU code that
        # replaces its own solver class by this one does: launches and copies.
        dict(name="mac_64_host", kind="solve", sys="mac", m=64, n=64, box="square", mixed=False, krylov=False, host=True),
        # A small ragged FEM projection of the channel, plain FP64.
        dict(name="fem_193x144", kind="solve", sys="fem", m=193, n=144, box="channel", mixed=False, krylov=False, host=False),
        # The rotor's MAC projection at its production size, mixed precision.
        dict(name="mac_1024_mixed", kind="solve", sys="mac", m=1024, n=1024, box="square", mixed=True, krylov=False, host=False),
        # A ragged MAC projection with conjugate gradients around the V-cycle.
        dict(name="mac_1501x997_krylov", kind="solve", sys="mac", m=1501, n=997, box="square", mixed=True, krylov=True, host=False),
        # The standalone MAC benchmark's size, plain FP64.
        dict(name="mac_4096", kind="solve", sys="mac", m=4096, n=4096, box="square", mixed=False, krylov=False, host=False),
        # The flag's FEM projection: cells three times as wide as high.
        dict(name="fem_2048_channel_mixed", kind="solve", sys="fem", m=2048, n=2048, box="channel", mixed=True, krylov=False, host=False),
        # ftest's default resolution: every kernel is small.
        dict(name="spin_128", kind="steps", scene="spin", m=128, bodies=1, mixed=False, guess=0, steps=10),
        # The rotor at the resolution of the published simulations.
        dict(name="spin_1024", kind="steps", scene="spin", m=1024, bodies=1, mixed=False, guess=0, steps=4),
        # 32 bodies settling on 1024 x 2048: many objects, plain FP64.
        dict(name="sediment_1024", kind="steps", scene="sediment", m=1024, bodies=32, mixed=False, guess=0, steps=4),
        # The headline benchmark: the literal 2048 x 2048 flag, FP32 V-cycles
        # and the quadratically extrapolated warm start.
        dict(name="flag_2048_mixed", kind="steps", scene="flag", m=2048, bodies=1, mixed=True, guess=2, steps=4),
        # The network on the grid of a 4096 x 4096 solve restricted by 8.
        dict(name="unet_infer_512", kind="infer", batch=1, H=512, W=512, base=32),
        # Its training on the flag's captured samples: batch 8 at 256 x 256.
        dict(name="unet_train_256", kind="train", batch=8, H=256, W=256, base=32),
    ]


def _log_size(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "steps", "steps", "unet"])
    if kind == "solve":
        box = rng.choice(["square", "square", "channel"])
        m = _log_size(rng, 64, 3000)
        if box == "channel":
            # the periodic direction has to halve down to a few rows
            n = rng.choice([4, 5, 6, 7, 9]) << rng.randint(4, 8)
            m = max(64, min(m, 2 * n))
        else:
            n = max(64, min(3000, int(m * rng.uniform(0.5, 2.0))))
        return dict(kind=kind, sys=rng.choice(["mac", "fem"]), m=m, n=n, box=box, mixed=rng.random() < 0.5,
                    krylov=rng.random() < 0.25, host=m * n < 300000 and rng.random() < 0.3)
    if kind == "steps":
        scene = rng.choice(["spin", "sediment", "flag"])
        if scene == "spin":
            m, bodies = _log_size(rng, 64, 1024), 1
        elif scene == "sediment":
            m, bodies = _log_size(rng, 384, 900), rng.randint(4, 24)
        else:
            m, bodies = rng.choice([768, 896, 1024, 1152, 1280, 1536, 1792]), 1
        return dict(kind=kind, scene=scene, m=m, bodies=bodies, mixed=rng.random() < 0.4, guess=rng.choice([0, 0, 1, 2]),
                    steps=rng.randint(2, 4))
    H, W = _log_size(rng, 64, 768, 16), _log_size(rng, 64, 768, 16)
    if rng.random() < 0.6:
        return dict(kind="infer", batch=rng.randint(1, 4), H=H, W=W, base=rng.choice([16, 32]))
    return dict(kind="train", batch=rng.randint(1, 8), H=min(H, 256), W=min(W, 256), base=rng.choice([16, 32]))


# ---------------------------------------------------------------------------
# Pressure solves

def _problem(case, seed):
    """The ghosted density (n+4, m+4) and the right-hand side of a solve."""
    m, n = case["m"], case["n"]
    box = CHANNEL if case["box"] == "channel" else SQUARE
    circ = workloads.circles(seed, box=box)
    rho = workloads.circle_density(m, n, circ, box=box, device="cuda")
    fem, channel = case["sys"] == "fem", case["box"] == "channel"
    if channel:
        rho[:2], rho[n + 2:] = rho[n:n + 2].clone(), rho[2:4].clone()
    mb, nb = (m + 1, n if channel else n + 1) if fem else (m, n)
    b = workloads.blob_divergence(mb, nb, seed, box=box, device="cuda")
    if fem and channel:
        b[:, -1] = 0  # the fixed column
    return rho.contiguous(), b.contiguous()


def _prepare_solve(case, seed):
    channel = case["box"] == "channel"
    box = CHANNEL if channel else SQUARE
    rho, b = _problem(case, seed)
    s = capi.MGSolver(capi.SYS_FEM if case["sys"] == "fem" else capi.SYS_MAC, case["m"], case["n"], *box,
                      y_prd=channel, zpr=channel)
    if case["krylov"]:
        s.set_krylov()
    state = dict(solver=s, host=case["host"], singular=not channel,
                 precision=capi.PREC_MIXED if case["mixed"] else capi.PREC_FP64)
    if case["host"]:
        state.update(rho=rho.cpu().numpy(), b=b.cpu().numpy())
    else:
        state.update(rho=rho, b=b, z=torch.empty_like(b), stream=torch.cuda.ExternalStream(s.stream()))
    return state


def _run_solve(state):
    s = state["solver"]
    if state["host"]:
        z = np.zeros_like(state["b"])
        s.set_density(state["rho"])
        s.solve(state["b"], z, precision=state["precision"])
        # with walls all round the pressure is defined up to a constant
        return z - z.mean() if state["singular"] else z
    z = state["z"]
    with torch.cuda.stream(state["stream"]):
        z.zero_()
        s.set_density_device(state["rho"].data_ptr())
        s.solve_device(state["b"].data_ptr(), z.data_ptr(), precision=state["precision"])
        return z - z.mean() if state["singular"] else z


def _mac_apply(case, rho):
    """z -> -A z of the MAC system (positive definite on the range)."""
    m, n = case["m"], case["n"]
    channel = case["box"] == "channel"
    box = CHANNEL if channel else SQUARE
    xx, yy = ((box[1] - box[0]) / m) ** -2, ((box[3] - box[2]) / n) ** -2
    ir = 1.0 / rho
    ex = xx * (0.5 * ir[2:n + 2, 2:m + 3] + 0.5 * ir[2:n + 2, 1:m + 2])
    ey = yy * (0.5 * ir[2:n + 3, 2:m + 2] + 0.5 * ir[1:n + 2, 2:m + 2])
    exi, right = ex[:, 1:m].contiguous(), 2 * ex[:, m]
    eyi, seam = ey[1:n].contiguous(), ey[0]
    diag = torch.zeros(n, m, dtype=torch.float64, device=rho.device)
    diag[:, 1:] += exi
    diag[:, :-1] += exi
    diag[1:] += eyi
    diag[:-1] += eyi
    if channel:
        diag[0] += seam
        diag[-1] += seam
        diag[:, -1] += right

    def apply(z):
        out = diag * z
        out[:, 1:] -= exi * z[:, :-1]
        out[:, :-1] -= exi * z[:, 1:]
        out[1:] -= eyi * z[:-1]
        out[:-1] -= eyi * z[1:]
        if channel:
            out[0] -= seam * z[-1]
            out[-1] -= seam * z[0]
        return out
    return apply, diag


def _fem_apply(case, rho):
    """z -> A z of the FEM system: bilinear elements, one per cell, the fixed
    right column of the channel left out."""
    m, n = case["m"], case["n"]
    channel = case["box"] == "channel"
    box = CHANNEL if channel else SQUARE
    dx, dy = (box[1] - box[0]) / m, (box[3] - box[2]) / n
    c = 1.0 / rho[2:n + 2, 2:m + 2]
    fm = (dx / dy + dy / dx) / 3
    hy, hx, fc = (dy / dx - 2 * dx / dy) / 6, (dx / dy - 2 * dy / dx) / 6, -(dx / dy + dy / dx) / 6
    nf = n if channel else n + 1

    def spread(cells):
        """Adds the (2, 2, n, m) corner values of the cells to their nodes."""
        out = torch.zeros(n + 1, m + 1, dtype=torch.float64, device=rho.device)
        for q in (0, 1):
            for p in (0, 1):
                out[q:q + n, p:p + m] += cells[q][p]
        if channel:
            out[0] += out[n]
        return out[:nf].contiguous()

    def apply(z):
        if channel:
            z = torch.cat([z, z[:1]])
            z[:, -1] = 0
        k = [[z[q:q + n, p:p + m] for p in (0, 1)] for q in (0, 1)]
        out = spread([[c * (fm * k[q][p] + hx * k[q][1 - p] + hy * k[1 - q][p] + fc * k[1 - q][1 - p])
                       for p in (0, 1)] for q in (0, 1)])
        if channel:
            out[:, -1] = 0
        return out
    diag = spread([[fm * c for _ in (0, 1)] for _ in (0, 1)])
    return apply, diag


def _exact_solve(case, seed):
    m, n = case["m"], case["n"]
    if m * n > 1600000:
        return None  # tens of thousands of iterations on millions of unknowns
    rho, b = _problem(case, seed)
    mac, singular = case["sys"] == "mac", case["box"] == "square"
    apply, diag = (_mac_apply if mac else _fem_apply)(case, rho)
    b = -b if mac else b
    x = torch.zeros_like(b)
    tiny = 1e-14 * b.norm()
    for _ in range(3):  # conjugate gradients, restarted from the true residual
        r = b - apply(x)
        if singular:
            r -= r.mean()
        y = r / diag
        p, ry = y.clone(), (r * y).sum()
        for it in range(20 * (m + n)):
            q = apply(p)
            a = ry / (p * q).sum()
            x += a * p
            r -= a * q
            y = r / diag
            new = (r * y).sum()
            p = y + (new / ry) * p
            ry = new
            if it % 50 == 49 and bool(r.norm() <= tiny):
                break
    x = x - x.mean() if singular else x
    return x.cpu().numpy() if case["host"] else x


# ---------------------------------------------------------------------------
# Time steps

def _prepare_steps(case, seed):
    m, rng = case["m"], np.random.default_rng(seed)
    prec = capi.PREC_MIXED if case["mixed"] else capi.PREC_FP64
    if case["scene"] == "spin":
        sim = capi.Simulation(m, m, ntrace=512, precision=prec)
        sim.add_simple_spin(r_scale=rng.uniform(0.7, 0.85), omega=rng.uniform(0.8, 1.2))
        box = SQUARE
    elif case["scene"] == "sediment":
        box = SEDIMENT
        sim = capi.Simulation(m, 2 * m, *box, visc=2e-3, ntrace=512, precision=prec)
        for o in workloads.sediment_bodies(seed=seed, count=case["bodies"]):
            if o["kind"] == "circle":
                sim.add_circle(o["cx"], o["cy"], o["r"], 1.0, o["rhos"], grav=o["grav"])
            else:
                sim.add_ellipse(o["cx"], o["cy"], o["r"], o["b"], o["theta"], 1.0, o["rhos"], grav=o["grav"])
    else:
        # aspect ratio 10, mass ratio 1, bending rigidity 0.1, Reynolds 100
        box, w = None, 0.1
        sim = capi.Simulation(m, m, *CHANNEL, visc=0.01, ntrace=0, precision=prec, y_prd=True, horiz_flow=1.0)
        sim.add_flag(0.0, 0.0, 1.0, w, 0.25 * w, 4 * 0.1 / w ** 3, 1.0 / w, perturb_v=rng.uniform(0.05, 0.3), ntrace=17)
    dt = sim.initialize()
    if box:
        sim.set_tracers(np.stack([rng.uniform(box[0], box[1], 512), rng.uniform(box[2], box[3], 512)], axis=1))
    sim.set_guess(case["guess"])
    out = {k: torch.empty(sim.nl, sim.ml, dtype=torch.float64, pin_memory=True).numpy() for k in ("u", "v", "p", "phi", "X", "Y")}
    return dict(sim=sim, dt=dt, steps=case["steps"], tracers=bool(box), out=out)


def _run_steps(state):
    sim = state["sim"]
    sim.step(state["dt"], state["steps"])
    out = {k: sim.get(k, out=v) for k, v in state["out"].items()}
    out["tracers"] = sim.tracers() if state["tracers"] else sim.object_tracers()
    return out


# ---------------------------------------------------------------------------
# The network

def _layers(base, levels=4):
    """(inputs, outputs, taps) of the network's convolutions in order."""
    c = [base << l for l in range(levels)]
    out = [(16, c[0], 9), (c[0], c[0], 9)]
    for l in range(1, levels):
        out += [(c[l - 1], c[l], 9), (c[l], c[l], 9)]
    for l in range(levels - 2, -1, -1):
        out += [(c[l + 1] + c[l], c[l], 9), (c[l], c[l], 9)]
    return out + [(c[0], 16, 1)]


def _network_inputs(case, seed):
    """He-uniform parameters (each layer's [tap][in][out] weights, then its
    biases) and images: a residual of unit variance, a reciprocal density, a
    zero channel; targets of unit variance on a mask that leaves some rows
    of padding out."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, W = case["batch"], case["H"], case["W"]
    parts = []
    for cin, cout, taps in _layers(case["base"]):
        parts += [(2 * torch.rand(taps * cin * cout, generator=g, device="cuda") - 1) * math.sqrt(6.0 / (taps * cin)),
                  0.02 * torch.randn(cout, generator=g, device="cuda")]
    x = torch.zeros(B, H, W, 3, device="cuda")
    x[..., 0] = torch.randn(B, H, W, generator=g, device="cuda")
    x[..., 1] = 1 / (1 + 2 * (torch.rand(B, H, W, generator=g, device="cuda") < 0.1).float())
    target = torch.randn(B, H, W, generator=g, device="cuda")
    valid = torch.ones(B, H, W, device="cuda")
    valid[:, H - 5:] = 0
    return torch.cat(parts), x, target * valid, valid


def _prepare_network(case, seed):
    params, x, target, valid = _network_inputs(case, seed)
    net = capi.UNet(4, case["base"])
    net.set_params(params.cpu().numpy())
    return dict(net=net, shape=(case["batch"], case["H"], case["W"]), train=case["kind"] == "train", x=x, target=target,
                valid=valid, out=torch.empty_like(target))


def _run_network(state):
    net, x = state["net"], state["x"]
    stream = torch.cuda.current_stream().cuda_stream
    if state["train"]:
        loss = net.train_step(*state["shape"], x.data_ptr(), state["target"].data_ptr(), state["valid"].data_ptr(), 2e-3,
                              stream)
        return dict(loss=loss, params=net.get_params())
    net.forward(*state["shape"], x.data_ptr(), state["out"].data_ptr(), stream)
    return state["out"]


def _exact_network(case, seed):
    import torch.nn.functional as F
    params, x, target, valid = (t.double() for t in _network_inputs(case, seed))
    params.requires_grad_(case["kind"] == "train")
    layers, at = [], 0
    for cin, cout, taps in _layers(case["base"]):
        k = 3 if taps == 9 else 1
        w = params[at:at + taps * cin * cout].reshape(k, k, cin, cout).permute(3, 2, 0, 1)
        at += taps * cin * cout
        layers.append((w, params[at:at + cout], k // 2))
        at += cout
    convs = iter(layers)

    def conv(h):
        w, bias, pad = next(convs)
        return F.relu(F.conv2d(h, w, bias, padding=pad)) if pad else F.conv2d(h, w, bias)
    with torch.set_grad_enabled(case["kind"] == "train"):
        h = F.pad(x, (0, 13)).permute(0, 3, 1, 2)
        skips = []
        for l in range(4):
            h = conv(conv(F.avg_pool2d(h, 2) if l else h))
            skips.append(h)
        for l in (2, 1, 0):
            h = conv(conv(torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), skips[l]], dim=1)))
        y = conv(h)[:, 0]
        if case["kind"] == "infer":
            return y
        loss = (valid * (y - target) ** 2).sum() / valid.sum()
        loss.backward()
    # Adam's first step: the bias-corrected moments are g and g^2
    g = params.grad
    return dict(loss=float(loss), params=(params.detach() - 2e-3 * g / (g.abs() + 1e-8)).cpu().numpy())


# ---------------------------------------------------------------------------

def prepare(case, seed):
    return {"solve": _prepare_solve, "steps": _prepare_steps}.get(case["kind"], _prepare_network)(case, seed)


def run(state):
    if "solver" in state:
        return _run_solve(state)
    return _run_steps(state) if "sim" in state else _run_network(state)


def exact(case, seed):
    """The solution by conjugate gradients in FP64, or the network in FP64. A
    simulation's step is some thirty coupled passes with no short restatement."""
    if case["kind"] == "steps":
        return None
    return _exact_solve(case, seed) if case["kind"] == "solve" else _exact_network(case, seed)


def work(case):
    """Inputs read once, outputs written once; the operations of the V-cycles
    (about nine from a zero start, five per warm-started projection, some 150
    operations per unknown of the finest level) or of the convolutions."""
    if case["kind"] == "solve":
        N = case["m"] * case["n"]
        return dict(bytes=8.0 * 3 * N, flops=9 * 150.0 * N)
    if case["kind"] == "steps":
        N = case["m"] * case["m"] * (2 if case["scene"] == "sediment" else 1)
        # velocity, pressure, density and the solids' reference map and level
        # set, read and written every step; the fields copied out at the end
        return dict(bytes=8.0 * N * (2 * 7 * case["steps"] + 6), flops=case["steps"] * N * (10 * 150.0 + 600))
    B, H, W = case["batch"], case["H"], case["W"]
    flops, pixels, at = 0.0, B * H * W, 0
    levels = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
    for (cin, cout, taps), l in zip(_layers(case["base"]), levels):
        flops += 2.0 * taps * cin * cout * (pixels >> (2 * l))
        at += taps * cin * cout + cout
    if case["kind"] == "infer":
        return dict(bytes=4.0 * (4 * pixels + at), flops=flops)
    return dict(bytes=4.0 * (5 * pixels + 6 * at), flops=3 * flops)

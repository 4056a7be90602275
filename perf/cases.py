"""Work that users of the framework have it do, as cases to be timed: one pass each through the public entry points.

A case is a dict of plain values; ``kind`` names the path:

emulate  one iceflow update in emulated mode: the 16-layer network over the whole domain, its velocities and the
         derived 2-D fields (processes.iceflow.update)
train    one physics-informed Adam step of the network on a batch of windows of the domain (emulator.train_step)
solve    a plain solve of the flow from the previous time step's velocities (DeviceAdamSolver.solve)
energy   the energy and its gradient with respect to the velocities, as a loss under autograd (energy.iceflow_energy)
mass     surface mass balance and thickness transport of one time step (processes.smb_simple.update, thk.update)
vert     the vertical velocity (processes.vert_flow.update)
invert   the inner loop of a thickness inversion: the emulator forward, the observation costs with their gradients and
         the emulator's adjoint down to the thickness (CNN.forward / backward, kernels.assim_*)

Glaciers are the synthetic valley of the benchmark (per-cell rate factor and sliding coefficient), made on the GPU."""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from igm_b200 import _lib as L
from igm_b200 import kernels as K
from igm_b200.cnn import CNN
from igm_b200.config import default_cfg
from igm_b200.emulator import EmulatorOptimizer, train_step
from igm_b200.energy import iceflow_energy
from igm_b200.processes import iceflow, smb_simple, thk, vert_flow
from igm_b200.solver import DeviceAdamSolver
from igm_b200.state import State
from igm_b200.vertical import compute_levels, compute_zeta_dzeta, define_vertical_weight

DX = 50.0
LAYERS, FILTERS, ALPHA = 16, 32, 0.01
SCALES = [1 / 300.0, 1 / 3000.0, 1 / 100.0, 10.0, 1 / 50.0]  # of the network's inputs thk, usurf, arrhenius, slidingco, dx
OUTPUT_SCALE = 50.0
FIELDS = ("thk", "usurf", "arrhenius", "slidingco")
ELA = (0.009, 0.009, 2900.0, 2.0)  # ablation and accumulation gradients, equilibrium line altitude, largest accumulation
LR, CLIPNORM, EPS = 2e-5, 1.0, 1e-7


def listed():
    return [
        # a time step of a small glacier: latency and launches count
        dict(name="emulate_100", kind="emulate", ny=100, nx=100, nz=10),
        # a time step of the benchmark's glacier
        dict(name="emulate_1000", kind="emulate", ny=1000, nx=1000, nz=10),
        # the large domain: 4096 x 4096 with 16 levels
        dict(name="emulate_4096", kind="emulate", ny=4096, nx=4096, nz=16),
        # training from scratch: batches of small windows
        dict(name="train_8x64", kind="train", ny=1000, nx=1000, nz=10, batch=8, h=64, w=64),
        # retraining during a run: the whole domain as one window
        dict(name="train_1000", kind="train", ny=1000, nx=1000, nz=10, batch=1, h=1000, w=1000),
        # the plain method on the 100 x 100 glacier, ten optimiser iterations
        dict(name="solve_100", kind="solve", ny=100, nx=100, nz=10, iterations=10),
        # the plain method (and the emulator's judge) on the benchmark's glacier
        dict(name="solve_1000", kind="solve", ny=1000, nx=1000, nz=10, iterations=10),
        # an own loss on the energy, on a real domain's odd extent
        dict(name="energy_701x1003", kind="energy", ny=701, nx=1003, nz=10, dtype="float32"),
        # the reference minimisation in double precision
        dict(name="energy_400_f64", kind="energy", ny=400, nx=400, nz=10, dtype="float64"),
        # mass balance and transport of one time step
        dict(name="mass_1000", kind="mass", ny=1000, nx=1000),
        # vertical velocity for the particles and the enthalpy
        dict(name="vert_1000", kind="vert", ny=1000, nx=1000, nz=10, method="kinematic"),
        # one inner iteration of a thickness inversion of a valley
        dict(name="invert_500x750", kind="invert", ny=500, nx=750, nz=10),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["emulate", "train", "solve", "energy", "mass", "vert", "invert"])
    c = dict(kind=kind, ny=size(64, 2048), nx=size(64, 2048), nz=rng.choice([5, 8, 10, 12, 16]))
    if kind == "train":
        c["batch"] = rng.choice([1, 1, 2, 4, 8])
        c["h"] = min(c["ny"], size(32, 1000 // c["batch"]))
        c["w"] = min(c["nx"], size(32, 1000))
    elif kind == "solve":
        c["ny"], c["nx"], c["iterations"] = min(c["ny"], 1400), min(c["nx"], 1400), rng.randint(1, 10)
    elif kind == "energy":
        c["dtype"] = rng.choice(["float32", "float32", "float64"])
        if c["dtype"] == "float64":
            c["ny"], c["nx"] = min(c["ny"], 700), min(c["nx"], 700)
    elif kind == "mass":
        del c["nz"]
    elif kind == "vert":
        c["method"] = rng.choice(["kinematic", "kinematic", "incompressibility"])
    elif kind == "invert":
        c["ny"], c["nx"] = min(c["ny"], 1000), min(c["nx"], 1000)
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _glacier(ny, nx, seed, dev):
    """The benchmark's valley mapped onto ny x nx cells of DX: a valley bed with noise, a tongue thinning downstream,
    rate factor and sliding coefficient log-uniform per cell, smoothed over 5 cells.  float32 fields [ny, nx]."""
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    x = torch.linspace(0, 10000.0, nx, device=dev, dtype=torch.float64)[None]
    y = torch.linspace(0, 10000.0, ny, device=dev, dtype=torch.float64)[:, None]

    def noise():
        return torch.rand(ny, nx, generator=g, device=dev, dtype=torch.float32)

    def smooth(a):
        return F.avg_pool2d(F.pad(a[None, None], (2, 2, 2, 2), mode="replicate"), 5, 1)[0, 0].contiguous()

    topg = (3000.0 - 0.1 * x + 0.002 * (y - 5000.0) ** 2).float() + 2.5 * torch.randn(ny, nx, generator=g, device=dev)
    h = (300.0 * (1 - ((y - 5000.0) / 2500.0) ** 2) * (1 - x / 10000.0)).clamp(min=0.0).float()
    h = h * (0.9 + 0.2 * smooth(noise()))
    return dict(topg=topg, thk=h, usurf=topg + h, arrhenius=smooth(20.0 * (150.0 / 20.0) ** noise()),
                slidingco=smooth(0.01 * 10.0 ** noise()))


def _velocities(g, nz, seed, dtype=torch.float32):
    """Velocities of a previous time step [nz, ny, nx]: down the valley, faster towards the surface and with the
    thickness, with some noise; zero off the ice."""
    dev = g["thk"].device
    r = torch.Generator(device=dev)
    r.manual_seed(int(seed) + 1)
    h = g["thk"]
    z = torch.linspace(0, 1, nz, device=dev)[:, None, None]
    ice = (h > 0).float()
    u = (5.0 + 60.0 * (h / 300.0) ** 2 * (0.4 + 0.6 * z) + 2.0 * torch.randn(nz, *h.shape, generator=r, device=dev)) * ice
    v = (2.0 + 4.0 * (h / 300.0) * z) * torch.randn(nz, *h.shape, generator=r, device=dev) * ice
    return u.to(dtype), v.to(dtype)


def _weights(nz, seed):
    """He-normal kernels and small biases in Keras order: 3x3 kernels [3, 3, cin, 32], the 1x1 head, each with its bias."""
    rng = np.random.default_rng(int(seed))
    out = []
    for i in range(LAYERS + 1):
        k, cin, cout = (1, FILTERS, 2 * nz) if i == LAYERS else (3, 5 if i == 0 else FILTERS, FILTERS)
        std = math.sqrt(2.0 / (k * k * cin))
        out.append(rng.normal(0, std, (k, k, cin, cout)).clip(-2 * std, 2 * std).astype(np.float32))
        out.append(rng.normal(0, 0.01, cout).astype(np.float32))
    return out


def _flat(weights):
    return np.concatenate([w.ravel() for w in weights])


def _network(nz, seed, dev):
    net = CNN(nb_layers=LAYERS, cin=5, nout=2 * nz, scales=SCALES, out_scale=OUTPUT_SCALE, alpha=ALPHA, device=dev)
    net.set_params(_flat(_weights(nz, seed)))
    return net


def _vertical(nz):
    levels = compute_levels(nz, 4.0)
    return levels, compute_zeta_dzeta(levels)[1], define_vertical_weight(nz, 4.0)


def _windows(case, seed):
    rng = np.random.default_rng(int(seed) + 2)
    return [(int(rng.integers(0, case["ny"] - case["h"] + 1)), int(rng.integers(0, case["nx"] - case["w"] + 1)))
            for _ in range(case["batch"])]


def _observations(g, seed):
    """Observed surface velocities with a tenth missing and thickness profiles on every 50th column."""
    h = g["thk"]
    r = torch.Generator(device=h.device)
    r.manual_seed(int(seed) + 3)
    nan = torch.full_like(h, float("nan"))
    ice = (h > 0).float()
    hole = torch.rand(h.shape, generator=r, device=h.device) < 0.1
    uobs = torch.where(hole, nan, 40.0 * (h / 300.0) * ice + torch.randn(h.shape, generator=r, device=h.device) * ice)
    vobs = torch.where(hole, nan, torch.randn(h.shape, generator=r, device=h.device) * ice)
    thkobs = nan.clone()
    thkobs[:, ::50] = h[:, ::50]
    return dict(uobs=uobs, vobs=vobs, thkobs=thkobs, dens=torch.ones_like(h), mask=ice)


def prepare(case, seed):
    dev = torch.device("cuda")
    kind, ny, nx, nz = case["kind"], case["ny"], case["nx"], case.get("nz", 10)
    g = _glacier(ny, nx, seed, dev)
    levels, dz, weight = _vertical(nz)
    fields = [g[k] for k in FIELDS]
    s = dict(kind=kind, case=case)
    if kind == "emulate":
        cfg = default_cfg({"iceflow": {"method": "emulated", "numerics": {"Nz": nz},
                                       "emulator": {"retrain_freq": 0, "pretrained": False, "input_scales": SCALES,
                                                    "output_scale": OUTPUT_SCALE}}})
        st = State()
        for k, v in g.items():
            setattr(st, k, v)
        st.dx, st.it, st.t = DX, 1, 0.0
        iceflow.initialize(cfg, st)
        st.iceflow_model.set_params(_flat(_weights(nz, seed)))
        s.update(cfg=cfg, st=st)
    elif kind == "train":
        s.update(net=_network(nz, seed, dev), fields=fields, dz=dz, phys=L.make_physics(), windows=_windows(case, seed),
                 opt=EmulatorOptimizer(LR, EPS, CLIPNORM))
    elif kind == "solve":
        U, V = _velocities(g, nz, seed)
        s.update(solver=DeviceAdamSolver(lr=1.0), U=U, V=V, fields=fields, dz=dz, phys=L.make_physics())
    elif kind == "energy":
        dt = getattr(torch, case["dtype"])
        U, V = _velocities(g, nz, seed, dt)
        s.update(U=U.requires_grad_(True), V=V.requires_grad_(True), fields=[f.to(dt) for f in fields], dz=dz)
    elif kind == "mass":
        cfg = default_cfg({"smb_simple": {"update_freq": 0.0, "array": [["time", "gradabl", "gradacc", "ela", "accmax"],
                                                                        [0.0, *ELA], [1e6, *ELA]]}})
        st = State()
        for k, v in g.items():
            setattr(st, k, v)
        U, V = _velocities(g, 2, seed)
        st.ubar, st.vbar = U[1].contiguous(), V[1].contiguous()
        st.dx, st.it, st.t, st.dt = DX, 0, 0.0, 0.1
        smb_simple.initialize(cfg, st)
        s.update(cfg=cfg, st=st)
    elif kind == "vert":
        cfg = default_cfg({"iceflow": {"numerics": {"Nz": nz}}, "vert_flow": {"method": case["method"]}})
        st = State()
        for k, v in g.items():
            setattr(st, k, v)
        st.U, st.V = _velocities(g, nz, seed)
        st.dx, st.vert_weight = DX, weight
        s.update(cfg=cfg, st=st)
    else:
        net = _network(nz, seed, dev)
        obs = _observations(g, seed)
        p = L.AssimParams()
        p.velsurfobs_std, p.thkobs_std, p.regu_thk, p.gamma, p.aniso_factor = 1.0, 3.0, 10.0, 1e-8, 0.2
        p.n_vel = float((~torch.isnan(obs["uobs"])).sum().item() * 2)
        p.n_thk = float((~torch.isnan(obs["thkobs"])).sum().item())
        p.penalty, p.icemask_cost, p.mask_velsurf = 1, 1, 1
        dU = torch.zeros(1, nz, ny, nx, device=dev)
        flow = K.assim_flow_direction(*[v[-1].contiguous() for v in _velocities(g, nz, seed)])
        s.update(net=net, g=g, fields=fields, obs=obs, params=p, buf=net.buffers(1, ny, nx, train=True), dU=dU,
                 dV=torch.zeros_like(dU), grad=torch.empty(1, 1, ny, nx, device=dev), flow=flow)
    return s


def run(s):
    kind = s["kind"]
    if kind == "emulate":
        st = s["st"]
        iceflow.update(s["cfg"], st)
        return dict(U=st.U, V=st.V, ubar=st.ubar, vbar=st.vbar, uvelbase=st.uvelbase, vvelbase=st.vvelbase,
                    uvelsurf=st.uvelsurf, vvelsurf=st.vvelsurf)
    if kind == "train":
        c, net = s["case"], s["net"]
        terms = train_step(net, s["fields"], DX, s["windows"], c["h"], c["w"], s["dz"], s["phys"], LR, s["opt"])
        return dict(terms=terms, grads=net.grads, params=net.params)
    if kind == "solve":
        U, V, costs = s["solver"].solve(s["U"], s["V"], *s["fields"], DX, s["dz"], nbitmax=s["case"]["iterations"],
                                        phys=s["phys"], early_stopping=False)
        return dict(U=U, V=V, costs=costs)
    if kind == "energy":
        U, V = s["U"], s["V"]
        cost = iceflow_energy(U, V, *s["fields"], DX, s["dz"])
        dU, dV = torch.autograd.grad(cost, [U, V])
        return dict(cost=cost, dU=dU, dV=dV)
    if kind == "mass":
        st = s["st"]
        smb_simple.update(s["cfg"], st)
        thk.update(s["cfg"], st)
        return dict(smb=st.smb, thk=st.thk, usurf=st.usurf, lsurf=st.lsurf, divflux=st.divflux)
    if kind == "vert":
        vert_flow.update(s["cfg"], s["st"])
        return dict(W=s["st"].W)
    net, g, o, buf = s["net"], s["g"], s["obs"], s["buf"]
    ny, nx = g["thk"].shape
    net.prepare_input(s["fields"], DX, [(0, 0)], ny, nx, buf)
    U, V = net.forward(buf, 1, ny, nx, keep_acts=True)
    costs, g_thk, _, _ = K.assim_cost_grad(g["thk"], g["usurf"], U[0, -1], V[0, -1], o["uobs"], o["vobs"], o["thkobs"],
                                           o["dens"], o["mask"], s["flow"], DX, s["params"], g_u=s["dU"][0, -1],
                                           g_v=s["dV"][0, -1])
    net.backward(buf, 1, ny, nx, s["dU"], s["dV"], field_grad=s["grad"], param_grads=False)
    return dict(U=U, V=V, costs=costs, dcost_dthk=g_thk, dcost_dvel=[s["dU"][0, -1], s["dV"][0, -1]],
                emulator_dthk=s["grad"])


def work(case):
    kind, px, nz = case["kind"], case["ny"] * case["nx"], case.get("nz", 10)
    params = 9 * 5 * FILTERS + FILTERS + (LAYERS - 1) * (9 * FILTERS * FILTERS + FILTERS) + (FILTERS + 1) * 2 * nz
    first, hidden, head = 2 * 9 * 5 * FILTERS, (LAYERS - 1) * 2 * 9 * FILTERS * FILTERS, 2 * FILTERS * 2 * nz
    cell = 190 * nz + 150  # operations of the energy of a column, counted in its formula; its gradient about twice that
    if kind == "emulate":  # reads the four fields, writes U, V and six 2-D fields
        return dict(bytes=px * 4.0 * (4 + 2 * nz + 6) + 4 * params, flops=px * float(first + hidden + head))
    if kind == "train":  # reads the windows, the parameters and moments; writes gradients, parameters and moments
        px = case["batch"] * case["h"] * case["w"]
        return dict(bytes=px * 16.0 + 28 * params, flops=px * float(2 * first + 3 * hidden + 3 * head + 3 * cell))
    if kind == "solve":  # an iteration reads and writes U, V and the four moments
        n = case["iterations"]
        return dict(bytes=px * n * 4.0 * (12 * nz + 4), flops=px * n * float(3 * cell + 24 * nz))
    if kind == "energy":
        e = 8 if case["dtype"] == "float64" else 4
        return dict(bytes=px * float(e) * (4 * nz + 4), flops=px * 3.0 * cell)
    if kind == "mass":  # reads thk, topg, usurf, ubar, vbar; writes smb, thk, usurf, lsurf, divflux
        return dict(bytes=px * 40.0, flops=px * 120.0)
    if kind == "vert":
        return dict(bytes=px * 4.0 * (3 * nz + 2), flops=px * 60.0 * nz)
    # reads the fields, the observations and the flow direction; writes U, V, the costs' and the emulator's gradients
    return dict(bytes=px * 4.0 * (4 + 7 + 2 * nz + 4), flops=px * float(2 * (first + hidden + head) + 150))


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------------
def _stag(a):
    return (a[..., 1:, 1:] + a[..., 1:, :-1] + a[..., :-1, 1:] + a[..., :-1, :-1]) / 4


def _dstag(a):
    dx, dy = (a[..., :, 1:] - a[..., :, :-1]) / DX, (a[..., 1:, :] - a[..., :-1, :]) / DX
    return (dx[..., 1:, :] + dx[..., :-1, :]) / 2, (dy[..., :, 1:] + dy[..., :, :-1]) / 2


def _terms64(U, V, h, s, A, c, nz):
    """Sums of the shear, sliding and gravity energies of the cells; U, V [B, nz, ny, nx], the fields [B, ny, nx]."""
    dz = torch.as_tensor(_vertical(nz)[1]).to(U)[None, :, None, None]

    def mid(a):
        return (a[:, 1:] + a[:, :-1]) / 2

    bx, by = _dstag(s - h)
    sx, sy = _dstag(s)
    Us, Vs, hs, cs = _stag(U), _stag(V), _stag(h), _stag(c)
    B = _stag(2.0 * A ** (-1.0 / 3.0))[:, None]
    (ux, uy), (vx, vy) = [[mid(d) for d in _dstag(w)] for w in (U, V)]
    lift = torch.where(cs > 0, 1.0, 0.01)[:, None] / (dz * hs.clamp(min=0.1)[:, None])
    uz, vz = (Us[:, 1:] - Us[:, :-1]) * lift, (Vs[:, 1:] - Vs[:, :-1]) * lift
    ux, uy = ux - uz * bx[:, None], uy - uz * by[:, None]
    vx, vy = vx - vz * bx[:, None], vy - vz * by[:, None]
    sr2 = 0.5 * (ux ** 2 + vy ** 2 + (ux + vy) ** 2 + 0.5 * (vx + uy) ** 2) + 0.25 * (uz ** 2 + vz ** 2)
    shear = hs * (B * dz * (sr2 + 1e-10) ** (-1.0 / 3.0) * sr2 / (4.0 / 3.0)).sum(1)
    ub, vb = Us[:, 0], Vs[:, 0]
    slide = cs * (ub ** 2 + vb ** 2 + 1e-20 + (ub * bx + vb * by) ** 2) ** (2.0 / 3.0) / (4.0 / 3.0)
    pull = 910.0 * 9.81e-6 * hs * (dz * (mid(Us) * sx[:, None] + mid(Vs) * sy[:, None])).sum(1)
    return torch.stack([shear.sum(), slide.sum(), pull.sum()])


def _net64(weights, fields, nz):
    x = torch.stack([f * k for f, k in zip([*fields, torch.full_like(fields[0], DX)], np.float32(SCALES).astype(float))], 1)
    for i in range(LAYERS + 1):
        w, b = weights[2 * i].permute(3, 2, 0, 1), weights[2 * i + 1]
        x = F.conv2d(x, w, b, padding=w.shape[-1] // 2)
        if i < LAYERS:
            x = F.leaky_relu(x, ALPHA)
    return x[:, :nz] * OUTPUT_SCALE, x[:, nz:] * OUTPUT_SCALE


def _limited(a):
    """Superbee slopes along the last axis of the cells 1 .. n - 2 of a."""
    p, m = (a[..., 2:] - a[..., 1:-1]) / DX, (a[..., 1:-1] - a[..., :-2]) / DX

    def pick(x, y, smaller):
        same, less = x * y > 0, x.abs() < y.abs()
        return torch.where(same, torch.where(less == smaller, x, y), 0.0)

    return pick(pick(p, 2 * m, True), pick(m, 2 * p, True), False)


def _flux(u, h, dt):
    """Upwind fluxes through the n + 1 faces along the last axis, cells outside empty."""
    f = F.pad((u[..., 1:] + u[..., :-1]) / 2, (1, 1))
    f[..., 0], f[..., -1] = u[..., 0], u[..., -1]
    a = F.pad(h, (2, 2))
    s = _limited(a)
    a = a[..., 1:-1]
    c = f * dt / DX
    left, right = a[..., :-1] + 0.5 * DX * (1 - c) * s[..., :-1], a[..., 1:] - 0.5 * DX * (1 + c) * s[..., 1:]
    return f * torch.where(f > 0, left, right)


def exact(case, seed):
    kind, ny, nx, nz = case["kind"], case["ny"], case["nx"], case.get("nz", 10)
    dev = _device()
    if ny * nx > 2_500_000 or case.get("method") == "incompressibility":
        return None
    g = {k: v.double() for k, v in _glacier(ny, nx, seed, dev).items()}
    weights = [torch.as_tensor(w).to(dev).double() for w in _weights(nz, seed)] if kind in ("emulate", "train", "invert") else None
    if kind == "invert":  # the costs of the 16-bit network's velocities have no such value of their own
        with torch.no_grad():
            U, V = _net64(weights, [g[k][None] for k in FIELDS], nz)
        return dict(U=U, V=V, costs=None, dcost_dthk=None, dcost_dvel=None, emulator_dthk=None)
    if kind == "emulate":
        ice = g["thk"] > 0
        with torch.no_grad():
            U, V = [torch.where(ice, v[0], 0.0) for v in _net64(weights, [g[k][None] for k in FIELDS], nz)]
        w = torch.as_tensor(_vertical(nz)[2]).to(U)
        return dict(U=U, V=V, ubar=(U * w).sum(0), vbar=(V * w).sum(0), uvelbase=U[0], vvelbase=V[0], uvelsurf=U[-1],
                    vvelsurf=V[-1])
    if kind == "train":
        h, w = case["h"], case["w"]
        f = [torch.stack([g[k][y:y + h, x:x + w] for y, x in _windows(case, seed)]) for k in FIELDS]
        for v in weights:
            v.requires_grad_(True)
        terms = _terms64(*_net64(weights, f, nz), *f, nz)
        grads = torch.autograd.grad(terms.sum() / (case["batch"] * (h - 1) * (w - 1)), weights)
        new = []
        for v, d in zip(weights, grads):  # the first Adam step of the clipped gradient
            d = d * (CLIPNORM / max(float(d.norm()), CLIPNORM))
            new.append(v.detach() - LR * d / (d.abs() + EPS / math.sqrt(1 - 0.999)))
        return dict(terms=terms.detach(), grads=torch.cat([d.reshape(-1) for d in grads]),
                    params=torch.cat([v.reshape(-1) for v in new]))
    if kind == "energy":
        dt = getattr(torch, case["dtype"])
        U, V = [v.double().requires_grad_(True) for v in _velocities(_glacier(ny, nx, seed, dev), nz, seed, dt)]
        cost = _terms64(U[None], V[None], *[g[k][None] for k in FIELDS], nz).sum() / ((ny - 1) * (nx - 1))
        dU, dV = torch.autograd.grad(cost, [U, V])
        return dict(cost=cost.detach(), dU=dU, dV=dV)
    if kind == "solve":
        U, V = [v.double() for v in _velocities(_glacier(ny, nx, seed, dev), nz, seed)]
        m, v2, costs = [0.0, 0.0], [0.0, 0.0], []
        for t in range(1, case["iterations"] + 1):
            U.requires_grad_(True)
            V.requires_grad_(True)
            cost = _terms64(U[None], V[None], *[g[k][None] for k in FIELDS], nz).sum() / ((ny - 1) * (nx - 1))
            costs.append(float(cost.detach()))
            step = math.sqrt(1 - 0.999 ** t) / (1 - 0.9 ** t)
            new = []
            for i, (x, d) in enumerate(zip((U, V), torch.autograd.grad(cost, [U, V]))):
                m[i] = m[i] + (d - m[i]) * 0.1
                v2[i] = v2[i] + (d * d - v2[i]) * 0.001
                new.append(x.detach() - m[i] * step / (v2[i].sqrt() + 1e-7))
            U, V = new
        ice = g["thk"] > 0
        return dict(U=torch.where(ice, U, 0.0), V=torch.where(ice, V, 0.0), costs=np.array(costs))
    if kind == "vert":
        U, V = [v.double() for v in _velocities(_glacier(ny, nx, seed, dev), nz, seed)]
        levels, _, weight = [torch.as_tensor(a).to(U) for a in _vertical(nz)]
        up = g["thk"] * (levels - levels[0])[:, None, None]
        mean = weight.cumsum(0)
        qx, qy = [(v * weight).cumsum(0) / mean * up for v in (U, V)]

        def faces(a, out):  # values between the cells of the last axis, at the two ends by ``out``
            return torch.cat([out(a[..., :1], a[..., 1:2]), (a[..., 1:] + a[..., :-1]) / 2, out(a[..., -1:], a[..., -2:-1])], -1)

        def slope(a, out):
            return faces(a, out).diff(dim=-1) / DX

        def line(a, b):
            return 1.5 * a - 0.5 * b

        z = g["topg"] + up
        W = -(slope(qx, lambda a, b: a) + slope(qy.mT, lambda a, b: a).mT)
        return dict(W=W + U * slope(z, line) + V * slope(z.mT, line).mT)
    U, V = [v[1].double() for v in _velocities(_glacier(ny, nx, seed, dev), 2, seed)]
    d = g["usurf"] - ELA[2]
    smb = (d * torch.where(d < 0, ELA[0], ELA[1])).clamp(-100.0, ELA[3])
    qx, qy = _flux(U, g["thk"], 0.1), _flux(V.T, g["thk"].T, 0.1).T
    div = (qx[:, 1:] - qx[:, :-1]) / DX + (qy[1:] - qy[:-1]) / DX
    h = (g["thk"] + 0.1 * (smb - div)).clamp(min=0.0)
    low = torch.maximum(g["topg"], -0.910 * h)
    return dict(smb=smb, thk=h, usurf=low + h, lsurf=low, divflux=div)

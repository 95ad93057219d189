"""The work that users of this framework have it do, as measurable cases.

``listed()`` names the cases, ``draw`` makes more of the same ranges,
``prepare`` builds what a driver holds before the call, ``run`` is one pass
through the public entry points, ``work`` the bytes and operations that the
pass cannot do without, and ``exact`` the same outputs from a plain torch
restatement of the equations in 64 bits (no code of this package).

Kinds of case (``kind``):

* ``step``      one timestep of a resident state: ``Simulation.step`` and the
                ``energy`` record that the driver writes after it
* ``hosted``    a Fortran driver's round trip: upload the host arrays, step,
                download them
* ``conduct``   the RKL2 conduction operator alone, on a resident energy that
                the driver has just written
* ``ensemble``  one graph launch (six steps) of many uneven members
* ``train``     one training step of the conduction network (forward,
                backward, Adam)
* ``forward``   the conduction network on the windows that tile a grid

Decks (``deck``): ``vortex`` (resistive Orszag-Tang, periodic), ``blast``
(ideal, periodic), ``walls`` (arcade with hot spots between z walls, gravity,
anomalous resistivity, conduction), ``ions`` (partially ionised vortex with
Cowling resistivity), ``arcade`` (the conduction deck).
"""
import math

import numpy as np
import torch

from lare3d_b200 import abi, decks, ensemble, gpu, surrogate
from lare3d_b200.grid import grid as make_grid

STATE = ("rho", "energy", "vx", "vy", "vz", "bx", "by", "bz")
PERIODIC, USER = abi.BC_PERIODIC, abi.BC_USER
PRECISION = {"fp64": gpu.FP64, "fp32": gpu.FP32, "exact64": gpu.EXACT64}
GAMMA = 5.0 / 3.0


def listed():
    return [
        # production: the benchmark grid of a resistive run, in each precision
        dict(name="step_vortex_256_fp64", kind="step", deck="vortex", precision="fp64", nx=256, ny=256, nz=256),
        dict(name="step_vortex_256_fp32", kind="step", deck="vortex", precision="fp32", nx=256, ny=256, nz=256),
        # an ordinary desk-size ideal run (the 64^3 blast)
        dict(name="step_blast_64_fp64", kind="step", deck="blast", precision="fp64", nx=64, ny=64, nz=64),
        # the smallest runs (set-up tests, parameter scans): launches and latency count
        dict(name="step_blast_24_fp32", kind="step", deck="blast", precision="fp32", nx=24, ny=24, nz=24),
        # a coronal box: ragged, z walls, gravity, anomalous resistivity and conduction in the step
        dict(name="step_walls_ragged_fp64", kind="step", deck="walls", precision="fp64", nx=187, ny=94, nz=141),
        # checking against the Fortran code: the bit-for-bit engine on the driver's own host arrays
        dict(name="hosted_vortex_exact64", kind="hosted", deck="vortex", precision="exact64", nx=96, ny=80, nz=121),
        # a chromospheric run: ionisation balance and Cowling resistivity
        dict(name="step_ions_80_fp64", kind="step", deck="ions", precision="fp64", nx=80, ny=80, nz=80),
        # conduction-dominated sub-steps, about fifty explicit limits long
        dict(name="conduct_256_fp32", kind="conduct", deck="arcade", precision="fp32", nx=256, ny=256, nz=256),
        dict(name="conduct_ragged_fp64", kind="conduct", deck="arcade", precision="fp64", nx=160, ny=129, nz=177),
        # a parameter study: many small members in one launch
        dict(name="ensemble_16_fp32", kind="ensemble", precision="fp32", members=16, n_min=24, n_max=64),
        # the learned conduction: its training, and its inference on a 128^3 grid
        dict(name="train_64_windows", kind="train", windows=64),
        dict(name="forward_128", kind="forward", nx=128, ny=128, nz=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["hosted", "conduct", "conduct", "ensemble", "train", "forward"])
    if kind == "ensemble":
        return dict(kind=kind, precision="fp32", members=rng.randint(2, 16), n_min=16, n_max=8 * rng.randint(3, 8))
    if kind == "train":
        return dict(kind=kind, windows=rng.randint(8, 64))
    if kind == "forward":
        return dict(kind=kind, nx=64 * rng.randint(1, 2), ny=64 * rng.randint(1, 2), nz=64 * rng.randint(1, 2))
    cap = {"step": 256 ** 3, "hosted": 110 ** 3, "conduct": 256 ** 3}[kind]
    deck = {"step": rng.choice(["vortex", "vortex", "blast", "blast", "walls", "ions"]), "hosted": "vortex",
            "conduct": "arcade"}[kind]
    if deck == "walls":
        cap = 136 ** 3
    if deck == "ions":
        cap = 80 ** 3
    if kind == "conduct":
        cap = 190 ** 3
    while True:
        n = _log_int(rng, 16, 256)
        nx, ny, nz = (max(12, min(384, int(n * rng.uniform(0.6, 1.6)))) for _ in range(3))
        if 14 ** 3 <= nx * ny * nz <= cap:
            break
    precision = rng.choice(["fp64", "fp32"])
    if kind == "hosted" or (kind == "step" and deck in ("vortex", "blast") and nx * ny * nz < 200 ** 3
                            and rng.random() < 0.2):
        precision = "exact64"
    return dict(kind=kind, deck=deck, precision=precision, nx=nx, ny=ny, nz=nz)


# ---------------------------------------------------------------------------
# Inputs.  Every 3-D array here is a tensor over Fortran indices -2..n+2 in
# each axis, stored [z][y][x]; element (i, j, k) is at [k + 2, j + 2, i + 2].

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Grid:
    """Metrics of a uniform box: d*b (cell widths), d*c (centre distances),
    and node and cell coordinates, each broadcastable and indexed from -2."""

    def __init__(self, n, hi, bcs, dev):
        self.n = n
        self.m = make_grid(n[0], n[1], n[2], (0.0, hi), (0.0, hi), (0.0, hi), bcs=bcs)
        shape = ((1, 1, -1), (1, -1, 1), (-1, 1, 1))
        self.db, self.dc, self.b, self.c = [], [], [], []
        for d, ax in enumerate("xyz"):
            def pad(v, lo, size):
                out = np.zeros(size)
                out[lo + 2:lo + 2 + len(v)] = v
                if lo == -1:
                    out[0] = v[0]
                out[lo + 2 + len(v):] = v[-1]
                return torch.from_numpy(out).to(dev).view(shape[d])
            size = n[d] + 5
            self.db.append(pad(self.m["d%sb" % ax], -1, size))
            self.dc.append(pad(self.m["d%sc" % ax], -1, size))
            self.b.append(pad(self.m[ax + "b"], -2, size))
            self.c.append(pad(self.m[ax + "c"], -1, size))


def _params(case):
    """Control values (names of lare_params) of a deck."""
    p = dict(gamma=GAMMA, visc1=0.1, visc2=0.5, dt_multiplier=0.8)
    deck = case.get("deck")
    if deck in ("vortex", "ions"):
        p.update(resistive_mhd=1, eta_background=1.0e-3, eta0=0.0, j_max=1.0e10)
    if deck == "ions":
        p.update(eos_number=abi.EOS_ION, cowling_resistivity=1, **decks.neutral_constants(abi.EOS_ION))
    if deck == "walls":
        p.update(resistive_mhd=1, eta_background=1.0e-4, eta0=1.0e-3, j_max=5.0, conduction=1, heat_flux_limiter=1,
                 flux_limiter=0.1, kappa_0=1.0e-4, zbc_min=USER, zbc_max=USER)
    if deck == "arcade":
        p.update(dt_multiplier=0.9, conduction=1, heat_flux_limiter=1, flux_limiter=0.1, kappa_0=1.0e-3,
                 kappa_perp_ratio=1.0e-6, zbc_min=USER, zbc_max=USER)
    return p


def _bcs(p):
    return [(p.get(a + "bc_min", PERIODIC), p.get(a + "bc_max", PERIODIC)) for a in "xyz"]


def _curl(g, A):
    """Face fields of the edge potential A (three tensors over -2..n+2, taken
    periodic): the circulation around each face over the face's area."""
    def back(a, ax):  # value at index - 1
        return torch.roll(a, 1, dims=2 - ax)
    out = []
    for d in range(3):
        e, f = (d + 1) % 3, (d + 2) % 3
        out.append((A[f] - back(A[f], e)) / g.db[e] - (A[e] - back(A[e], f)) / g.db[f])
    return out


def _inputs(case, seed):
    """(grid, params, state tensors, dt, gravity or None) of a grid case."""
    dev = _device()
    n = (case["nx"], case["ny"], case["nz"])
    p = _params(case)
    deck = case["deck"]
    g = _Grid(n, 2.0 * math.pi if deck in ("vortex", "ions") else 1.0, [b[1] for b in _bcs(p)], dev)
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    shape = (n[2] + 5, n[1] + 5, n[0] + 5)
    ones = torch.ones(shape, dtype=torch.float64, device=dev)
    sin, cos = torch.sin, torch.cos
    ph = rng.uniform(0.0, 2.0 * math.pi, 12)
    (xb, yb, zb), (xc, yc, zc) = g.b, g.c
    grav = None
    s = {}
    if deck in ("vortex", "ions"):
        s4 = 1.0 / math.sqrt(4.0 * math.pi)
        v0 = 1.0 if deck == "vortex" else 0.3
        if deck == "vortex":
            rho0, p0 = 25.0 / (36.0 * math.pi), 5.0 / (12.0 * math.pi)
            s["rho"] = rho0 * (1.0 + 0.1 * sin(xc + ph[0]) * cos(zc + ph[1])) * ones
            s["energy"] = p0 / ((GAMMA - 1.0) * s["rho"])
        else:
            T = (1.8 + 0.4 * sin(xc + ph[0]) * sin(yc + ph[1]) * cos(zc + ph[2])) * ones
            s["rho"] = (1.0 + 0.05 * cos(yc + ph[3])) * ones
            xi = _get_neutral(T, s["rho"], p)
            s["energy"] = (T * (2.0 - xi) + (1.0 - xi) * p["ionise_pot"] * (GAMMA - 1.0)) / (GAMMA - 1.0)
        s["vx"] = -v0 * sin(zb + ph[4]) * ones
        s["vy"] = v0 * sin(xb + ph[5]) * ones
        s["vz"] = v0 * sin(yb + ph[6]) * ones
        # a seeded random vector potential on the periodic lattice
        idx = [torch.arange(-2, n[d] + 3, device=dev) % n[d] for d in range(3)]
        A = []
        for _ in range(3):
            a = 1.0e-3 * (2.0 * torch.rand((n[2], n[1], n[0]), dtype=torch.float64, device=dev, generator=gen) - 1.0)
            A.append(a[idx[2]][:, idx[1]][:, :, idx[0]])
        db = _curl(g, A)
        s["bx"] = -sin(zc + ph[7]) * s4 + db[0]
        s["by"] = sin(2.0 * xc + ph[8]) * s4 + db[1]
        s["bz"] = sin(yc + ph[9]) * s4 + db[2]
        dt = 0.3 * min(2.0 * math.pi / k for k in n) / 2.0
    elif deck == "blast":
        c = rng.uniform(0.4, 0.6, 3)
        th, fi = math.acos(rng.uniform(-1.0, 1.0)), rng.uniform(0.0, 2.0 * math.pi)
        r2 = (xc - c[0]) ** 2 + (yc - c[1]) ** 2 + (zc - c[2]) ** 2
        k = 2.0 * math.pi
        s["rho"] = (1.0 + 0.1 * sin(k * yc + ph[0]) * cos(k * xc + ph[1])) * ones
        pres = (0.1 + 0.02 * sin(k * xc + ph[2]) * sin(k * zc + ph[3])) + 9.9 / (1.0 + torch.exp((r2 - 0.01) / 0.002))
        s["energy"] = pres / ((GAMMA - 1.0) * s["rho"])
        s["vx"] = 0.1 * sin(k * zb + ph[4]) * cos(k * xb + ph[5]) * ones
        s["vy"] = 0.1 * sin(k * xb + ph[6]) * cos(k * yb + ph[7]) * ones
        s["vz"] = 0.1 * sin(k * yb + ph[8]) * cos(k * zb + ph[9]) * ones
        s["bx"] = math.sin(th) * math.cos(fi) * ones
        s["by"] = math.sin(th) * math.sin(fi) * ones
        s["bz"] = math.cos(th) * ones
        dt = 0.3 * min(1.0 / k for k in n) / 5.0
    else:  # walls, arcade: B = curl(A_y e_y), A_y = cos(kx) exp(-kz); isobaric hot spots
        k = 2.0 * math.pi
        Ay = cos(k * xb + ph[0]) * torch.exp(-k * zb) * torch.ones_like(yc)
        zero = torch.zeros_like(Ay)
        up = torch.roll(Ay, 1, dims=0)
        up[0] = Ay[0] * math.exp(k * float(g.m["dzb"][0]))
        left = torch.roll(Ay, 1, dims=2)
        left[:, :, 0] = (cos(k * (xb[..., 0] - float(g.m["dxb"][0])) + ph[0]) * torch.exp(-k * zb[..., 0]))
        s["bx"] = -(Ay - up) / g.db[2]
        s["by"] = zero.clone()
        s["bz"] = (Ay - left) / g.db[0]
        T = ones.clone()
        amp = 10.0 if deck == "arcade" else 3.0
        sig = 8.0 / max(n)
        for _ in range(8):
            c = rng.uniform(0.0, 1.0, 3)
            c[2] = 0.2 + 0.6 * c[2]
            dx, dy = torch.abs(xc - c[0]), torch.abs(yc - c[1])
            dx, dy = torch.minimum(dx, 1.0 - dx), torch.minimum(dy, 1.0 - dy)
            T = T + amp * torch.exp(-dx * dx / (2 * sig * sig)) * torch.exp(-dy * dy / (2 * sig * sig)) * torch.exp(
                -(zc - c[2]) ** 2 / (2 * sig * sig))
        s["rho"] = 1.0 / T
        s["energy"] = 2.0 * T / (GAMMA - 1.0)
        v0 = 0.2 if deck == "walls" else 0.0
        wall = sin(math.pi * zb)
        s["vx"] = v0 * wall * sin(k * yb + ph[1]) * torch.ones_like(xb)
        s["vy"] = v0 * wall * sin(k * xb + ph[2]) * torch.ones_like(yb)
        s["vz"] = v0 * wall * sin(k * (xb + yb) + ph[3])
        dt = 0.1 * min(1.0 / k for k in n) / 4.0
        if deck == "walls":
            grav = np.full(n[2] + 4, 0.1)
    if case["precision"] == "fp32":  # the values that the engine will hold
        s = {q: v.to(torch.float32).to(torch.float64) for q, v in s.items()}
    return g, p, s, dt, grav


# ---------------------------------------------------------------------------
# What a driver holds before the call.

class _DeviceArray:
    """Memory of a context, which it keeps alive."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides,
                                         "typestr": typestr, "version": 3}


class _Fields:
    """Named device arrays of a context as tensors over their Fortran bounds
    ([z][y][x]).  The engine rotates some buffers, so the address is asked
    for on every use and the tensor made once per address."""

    def __init__(self, sim):
        self.sim, self.views, self.bounds = sim, {}, {}

    def __call__(self, name):
        ptr, sx, sxy, eb = self.sim.field_device(name)
        t = self.views.get((name, ptr))
        if t is None:
            lo, hi = self.bounds.setdefault(name, self.sim.field_bounds(name))
            a = ptr + eb * (lo[0] + sx * lo[1] + sxy * lo[2])
            shape = tuple(h - l + 1 for l, h in zip(lo[::-1], hi[::-1]))
            t = torch.as_tensor(_DeviceArray(self.sim, a, shape, (eb * sxy, eb * sx, eb), "<f%d" % eb), device="cuda")
            self.views[(name, ptr)] = t
        return t

    def state(self):
        return {k: self(k) for k in STATE}


def _bounded(t, lo, hi):
    """The part lo..hi (Fortran bounds, x first) of a tensor over -2..n+2."""
    return t[lo[2] + 2:hi[2] + 3, lo[1] + 2:hi[1] + 3, lo[0] + 2:hi[0] + 3]


def _deck(case, g, p, grav):
    n = (case["nx"], case["ny"], case["nz"])
    return decks.Deck(case["deck"], abi.default_params(**p), n[0], n[1], n[2], g.m, None, nsteps=1, grav=grav)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        ds = []
        for spec in _members(case, seed):
            g, p, s = _member(spec)
            d = _deck(spec[0], g, p, None)
            d.state = _host_state(g, s)
            ds.append(d)
        return dict(kind=kind, ens=ensemble.Ensemble(ds, precision=PRECISION[case["precision"]]))
    if kind in ("train", "forward"):
        return _prepare_network(case, seed)
    g, p, s, dt, grav = _inputs(case, seed)
    sim = gpu.simulation(_deck(case, g, p, grav), precision=PRECISION[case["precision"]])
    st = dict(kind=kind, sim=sim, step=0)
    if kind == "hosted":  # the driver's own arrays, in pinned memory
        n = (sim.nx, sim.ny, sim.nz)
        st["host"] = abi.State(*n, arrays={})
        st["pinned"] = []
        for name in STATE:
            lo, hi = abi.bounds(abi.STATE_KINDS[name], *n)
            t = _bounded(s[name], lo, hi).contiguous().cpu().pin_memory()
            st["pinned"].append(t)
            st["host"][name] = t.numpy().T
        sim.set_time(0.0, dt)
        sim.upload(st["host"])
        sim.boundary_conditions()
        sim.eta_calc()
        sim.download(st["host"])
        return st
    f = _Fields(sim)
    for name in STATE:
        v = f(name)
        v.copy_(_bounded(s[name], *sim.field_bounds(name)))
    torch.cuda.synchronize()
    if grav is not None:
        sim.upload_aux(grav=grav)
    sim.set_time(0.0, dt)
    sim.boundary_conditions()
    sim.eta_calc()
    if case["deck"] == "ions":
        sim.neutral_fraction()
        sim.perpendicular_resistivity()
    st["fields"] = f
    if kind == "conduct":
        st["stream"] = torch.cuda.ExternalStream(gpu.stream_of(sim))
        st["dt"] = _conduct_dt(_Exact(g, p, s, dt, grav))
        st["energy"] = f("energy").clone()
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind == "ensemble":
        ens = st["ens"]
        ens.launch(1)
        ens.sync()
        views = st.setdefault("fields", [_Fields(sim) for sim in ens.sims])
        return {k: torch.cat([f(k).reshape(-1) for f in views]) for k in STATE}
    if kind == "train":
        net = st["net"]
        net.train_step(st["bufs"], st["nb"], 5e-4)
        return dict(prediction=st["bufs"]["out"], loss=net.loss, gradients=net.g, weights=net.p)
    if kind == "forward":
        st["net"].forward(st["bufs"], st["nb"])
        return dict(prediction=st["bufs"]["out"])
    sim = st["sim"]
    if kind == "conduct":
        with torch.cuda.stream(st["stream"]):  # the driver's own energy, then the operator
            st["fields"]("energy").copy_(st["energy"])
        stages = sim.conduct_heat(st["dt"])
        return dict(energy=st["fields"]("energy"), stages=stages)
    st["step"] += 1
    if kind == "hosted":
        sim.upload(st["host"])
        t, dt = sim.step(st["step"])
        sim.download(st["host"])
        return dict(time=t, dt=dt, **{k: st["host"][k] for k in STATE})
    t, dt = sim.step(st["step"])
    return dict(time=t, dt=dt, account=np.array(sim.energy()), **st["fields"].state())


def work(case):
    kind = case["kind"]
    if kind == "train":
        return dict(bytes=_window_bytes(case["windows"], 24), flops=3.0 * _net_flops(case["windows"], 24))
    if kind == "forward":
        nb = (case["nx"] // 64) * (case["ny"] // 64) * (case["nz"] // 64)
        return dict(bytes=_window_bytes(nb, 72), flops=_net_flops(nb, 72))
    word = 4 if case["precision"] == "fp32" else 8
    if kind == "ensemble":  # on average; six steps a launch, 8 arrays in and out
        n = sum(spec[0]["nx"] ** 3 for spec in _members(case, 0))
        return dict(bytes=16.0 * word * n, flops=6.0 * 3000.0 * n)
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "conduct":  # energy in and out, rho and B in; about 13 stages
        return dict(bytes=6.0 * word * n, flops=13.0 * 110.0 * n)
    if kind == "hosted":  # the state over the host link and back, and the step
        return dict(bytes=48.0 * word * n, flops=3000.0 * n)
    flops = {"vortex": 3000.0, "blast": 2700.0, "walls": 4000.0, "ions": 9000.0}[case["deck"]]
    return dict(bytes=16.0 * word * n, flops=flops * n)


# ---------------------------------------------------------------------------
# The network: windows of features with the spread that the conduction deck
# gives them, and random weights of the trained ones' size.

def _members(case, seed):
    """One case a member: the kinds and edges of the study are the case's
    own, plasma beta and resistivity (log-uniform) come from the seed."""
    study = np.random.default_rng([case["members"], case["n_min"], case["n_max"]])
    rng = np.random.default_rng(int(seed) + 1)
    out = []
    for _ in range(case["members"]):
        deck = "blast" if study.random() < 0.5 else "vortex"
        n = int(study.integers(case["n_min"], case["n_max"] + 1))
        beta, eta = math.exp(rng.uniform(math.log(0.1), math.log(10.0))), math.exp(rng.uniform(math.log(1e-4), math.log(1e-2)))
        out.append((dict(kind="step", deck=deck, precision=case["precision"], nx=n, ny=n, nz=n), beta, eta,
                    int(rng.integers(1, 1 << 30))))
    return out


def _member(spec):
    """(grid, parameters, state tensors) of one member."""
    case, beta, eta, seed = spec
    g, p, s, _dt, _grav = _inputs(case, seed)
    p.update(resistive_mhd=1, eta_background=eta, eta0=0.0, j_max=1.0e10)
    beta0 = 0.2 if case["deck"] == "blast" else 2.2
    for k in ("bx", "by", "bz"):
        s[k] = (s[k] * math.sqrt(beta0 / beta)).to(torch.float32).to(torch.float64)
    return g, p, s


def _host_state(g, s):
    st = abi.State.zeros(*g.n)
    for k in STATE:
        st[k][...] = _bounded(s[k], *abi.bounds(abi.STATE_KINDS[k], *g.n)).cpu().numpy().T
    return st


def _net_flops(nb, win):
    return sum(2.0 * 27 * cin * cf * (win - 2 * l - 2) ** 3 * nb for l, (_p, _c, cin, cf) in enumerate(surrogate.LAYERS))


def _window_bytes(nb, win):  # seven bf16 features in, one FP32 prediction out
    return nb * (14.0 * win ** 3 + 4.0 * (win - 8) ** 3)


def _network_inputs(case, seed):
    """(nb, win, bf16 windows [nb, w, w, w, 16], targets [nb, (w - 8)^3])."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(int(seed) + 5)
    train = case["kind"] == "train"
    win = 24 if train else 72
    nb = case["windows"] if train else (case["nx"] // 64) * (case["ny"] // 64) * (case["nz"] // 64)
    u = torch.rand((nb, 3, 4), dtype=torch.float32, device=dev, generator=gen)
    ax = [torch.arange(win, dtype=torch.float32, device=dev).view(sh) / 64.0
          for sh in ((1, 1, 1, -1), (1, 1, -1, 1), (1, -1, 1, 1))]
    x = torch.zeros((nb, win, win, win, 16), dtype=torch.bfloat16, device=dev)
    pick = lambda a, b: u[:, a, b].view(-1, 1, 1, 1)  # noqa: E731
    r2 = sum((ax[d] - 0.2 - 0.5 * pick(d, 0)) ** 2 for d in range(3))
    T = 0.1 + torch.exp(-20.0 * r2) + 0.01 * torch.rand((nb, win, win, win), device=dev, generator=gen)
    rho = 0.1 / T
    ang = 6.2831853 * (ax[0] + pick(0, 1)) + 0.0 * r2
    for c, v in enumerate((T, rho, torch.cos(ang), 0.1 * pick(1, 1) + 0.0 * r2, torch.sin(ang))):
        x[..., c] = v.to(torch.bfloat16)
    for c, v in ((5, T), (6, rho)):
        x[..., c] = (256.0 * (v - x[..., c - 5].to(torch.float32))).to(torch.bfloat16)
    tgt = torch.randn((nb, (win - 8) ** 3), dtype=torch.float32, device=dev, generator=gen)
    return nb, win, x, tgt


def _prepare_network(case, seed):
    nb, win, x, tgt = _network_inputs(case, seed)
    train = case["kind"] == "train"
    net = surrogate.Network(seed=int(seed) % (1 << 31))
    bufs = net.buffers(nb, win, train)
    bufs["x"].copy_(x.reshape(-1))
    if train:
        bufs["tgt"].copy_(tgt.reshape(-1))
    else:
        net.pack()
    torch.cuda.synchronize()
    return dict(kind=case["kind"], net=net, bufs=bufs, nb=nb)


def _net_params(seed):
    """Random initial weights [27][cout][cin] in 32 bits, as the network takes them."""
    rng = np.random.default_rng(int(seed) % (1 << 31))
    W = []
    for l, (cin, cout, cin_r, _cf) in enumerate(surrogate.LAYERS):
        last = l == len(surrogate.LAYERS) - 1
        cout_r = 1 if last else cout
        w = np.zeros((27, cout, cin), np.float32)
        std = math.sqrt(2.0 / (27.0 * cin_r)) * (0.1 if last else 1.0)
        w[:, :cout_r, :cin_r] = (rng.standard_normal((27, cout_r, cin_r)) * std).astype(np.float32)
        W.append(torch.from_numpy(w).to(_device()))
    return W


def _taps(d):
    return [(t, slice(t // 9, t // 9 + d), slice(t // 3 % 3, t // 3 % 3 + d), slice(t % 3, t % 3 + d)) for t in range(27)]


def _exact_network(case, seed):
    nb, win, x, tgt = _network_inputs(case, seed)
    master = _net_params(seed)
    W = [w.to(torch.bfloat16).to(torch.float64) for w in master]
    W[3] = W[3][:, :1]
    acts = [x.to(torch.float64)]
    for l in range(4):
        d = win - 2 * l - 2
        cin = W[l].shape[2]
        y = torch.zeros((nb * d ** 3, W[l].shape[1]), dtype=torch.float64, device=x.device)
        for t, a, b, c in _taps(d):
            y += acts[l][:, a, b, c].reshape(-1, cin) @ W[l][t].T
        y = y.view(nb, d, d, d, -1)
        acts.append(torch.relu(y) if l < 3 else y)
    out = acts[4][..., 0].reshape(nb, -1)
    if case["kind"] == "forward":
        return dict(prediction=out.reshape(-1))
    err = out - tgt.to(torch.float64)
    loss = err.square().mean()
    dy = torch.zeros((nb, 16, 16, 16, 16), dtype=torch.float64, device=x.device)
    dy[..., 0] = (2.0 * err / err.numel()).view(nb, 16, 16, 16)
    W[3] = master[3].to(torch.bfloat16).to(torch.float64)
    grads = [None] * 4
    for l in (3, 2, 1, 0):
        d = win - 2 * l - 2
        cout, cin = W[l].shape[1], W[l].shape[2]
        flat = dy.reshape(-1, cout)
        gw = torch.stack([flat.T @ acts[l][:, a, b, c].reshape(-1, cin) for _t, a, b, c in _taps(d)])
        grads[l] = (gw, flat.sum(0))
        if l:
            dx = torch.zeros_like(acts[l])
            for t, a, b, c in _taps(d):
                dx[:, a, b, c] += (flat @ W[l][t]).view(nb, d, d, d, cin)
            dy = dx * (acts[l] > 0)
    g = torch.cat([torch.cat([gw.reshape(-1), gb]) for gw, gb in grads])
    # (Adam's first step is close to the sign of a gradient that 16-bit
    # activations give: the weights after it have no 64-bit value to go by)
    return dict(prediction=out.reshape(-1), loss=loss.reshape(1), gradients=g, weights=None)


# ---------------------------------------------------------------------------
# The timestep in 64 bits, in plain torch: the Lagrangian step with shock
# viscosity, resistivity and conduction, and the three Van Leer remap sweeps.

UNIT = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
TINY = 2.2250738585072014e-308


class _Box:
    """Views over an index box lo..hi (x first) of tensors over -2..n+2;
    ``B(a, o)`` is a shifted by the offset o."""

    def __init__(self, lo, hi):
        self.lo, self.hi = lo, hi

    def __call__(self, a, o=(0, 0, 0)):
        sl = []
        for d in (2, 1, 0):
            if a.shape[2 - d] == 1:
                sl.append(slice(None))
            else:
                sl.append(slice(self.lo[d] + o[d] + 2, self.hi[d] + o[d] + 3))
        return a[tuple(sl)]


def _off(*axes):
    """Offset with -1 along axes given as ~d and +1 along axes given as d."""
    o = [0, 0, 0]
    for d in axes:
        o[d if d >= 0 else ~d] += 1 if d >= 0 else -1
    return tuple(o)


CORNERS = [(i, j, k) for k in (0, 1) for j in (0, 1) for i in (0, 1)]


class _Exact:
    def __init__(self, g, p, s, dt, grav):
        self.g, self.n = g, g.n
        q = abi.default_params(**p)
        self.p = {k: getattr(q, k) for k, _t in q._fields_}
        self.bc = _bcs(self.p)
        self.per = [b == (PERIODIC, PERIODIC) for b in self.bc]
        self.dev = s["rho"].device
        self.shape = tuple(s["rho"].shape)
        for k, v in s.items():
            setattr(self, k, v.clone())
        self.cv = g.db[0] * g.db[1] * g.db[2]
        self.dt, self.time = dt, 0.0
        self.grav = torch.zeros((self.shape[0], 1, 1), dtype=torch.float64, device=self.dev)
        if grav is not None:
            self.grav[1:, 0, 0] = torch.from_numpy(grav).to(self.dev)
        self.pip = self.p["eos_number"] not in (0, abi.EOS_IDEAL)
        self.xi = torch.full_like(self.rho, self.p["xi_n"]) if self.pip else self.p["xi_n"]
        self.eta_perp = self.zeros()
        self.visc_tot = self.ohm_tot = 0.0
        self.boundary_conditions()
        self.eta_and_fluxes(False)
        if self.pip:
            self.xi = self.neutral_fraction(self.energy)
            self.perpendicular_resistivity()

    def zeros(self):
        return torch.zeros(self.shape, dtype=torch.float64, device=self.dev)

    def box(self, lo, hi):
        """lo, hi relative to 0 and n, one number or one per axis."""
        lo = (lo,) * 3 if isinstance(lo, int) else lo
        hi = (hi,) * 3 if isinstance(hi, int) else hi
        return _Box(lo, tuple(self.n[d] + hi[d] for d in range(3)))

    # -- ghost cells
    def fill(self, a, stag, mpi=True, user=True):
        """stag: 'c', 'n' or 'f' per axis."""
        for d in range(3):
            n, kind = self.n[d], stag[d]
            v = a.movedim(2 - d, 0)

            def put(i, j):
                if j is None:
                    v[i + 2] = 0.0
                else:
                    v[i + 2] = v[j + 2]
            if self.per[d]:
                if mpi:
                    pairs = {"c": ((n + 1, 1), (n + 2, 2), (-1, n - 1), (0, n)),
                             "n": ((n, 0), (n + 1, 1), (n + 2, 2), (-2, n - 2), (-1, n - 1)),
                             "f": ((n + 1, 1), (n + 2, 2), (-2, n - 2), (-1, n - 1), (0, n))}[kind]
                    for i, j in pairs:
                        put(i, j)
            elif user:
                if self.bc[d][0] == USER:
                    for i, j in {"c": ((0, 1), (-1, 2)), "n": ((-2, None), (-1, None), (0, None)),
                                 "f": ((-1, 1), (-2, 2))}[kind]:
                        put(i, j)
                if self.bc[d][1] == USER:
                    for i, j in {"c": ((n + 1, n), (n + 2, n - 1)), "n": ((n, None), (n + 1, None), (n + 2, None)),
                                 "f": ((n + 1, n - 1), (n + 2, n - 2))}[kind]:
                        put(i, j)

    def fill_b(self):
        self.fill(self.bx, "fcc")
        self.fill(self.by, "cfc")
        self.fill(self.bz, "ccf")

    def fill_v(self, vs):
        for v in vs:
            self.fill(v, "nnn")

    def boundary_conditions(self):
        self.fill_b()
        self.fill(self.energy, "ccc")
        self.fill(self.rho, "ccc")
        self.fill_v((self.vx, self.vy, self.vz))

    # -- partially ionised plasma
    def neutral_fraction(self, e):
        p, out = self.p, self.zeros()
        B = self.box(-1, 2)
        g1, ip = p["gamma"] - 1.0, p["ionise_pot"]
        e0, r0 = B(e), B(self.rho)
        t = g1 * torch.clamp((e0 - ip) / 2.0, min=TINY)
        dx = g1 * e0 - t
        live = torch.ones_like(t, dtype=torch.bool)
        xi = torch.zeros_like(t)
        for _ in range(100):
            dx = torch.where(live, dx / 2.0, dx)
            x = t + dx
            xa = _get_neutral(x, r0, p)
            fa = x - g1 * (e0 - (1.0 - xa) * ip) / (2.0 - xa)
            xi = torch.where(live, xa, xi)
            t = torch.where(live & (fa <= 0.0), x, t)
            live = live & ~((dx.abs() < 1e-8) | (fa.abs() < 1e-8))
            if not bool(live.any()):
                break
        B(out).copy_(xi)
        return out

    def perpendicular_resistivity(self):
        p = self.p
        B = self.box(0, 0)
        rv = sum(B(self.rho, o) * B(self.cv, o) for o in CORNERS) / sum(B(self.cv, o) for o in CORNERS)
        bx, by, bz = self.bx, self.by, self.bz
        bxv = 0.25 * (B(bx) + B(bx, _off(1)) + B(bz, _off(2)) + B(bz, _off(1, 2)))
        byv = 0.25 * (B(by) + B(by, _off(0)) + B(bz, _off(2)) + B(bz, _off(0, 2)))
        bzv = 0.25 * (B(bz) + B(bz, _off(0)) + B(bz, _off(1)) + B(bz, _off(0, 1)))
        tv = sum((B(self.energy, o) - (1.0 - B(self.xi, o)) * p["ionise_pot"]) / (2.0 - B(self.xi, o)) for o in CORNERS)
        tv = tv * (p["gamma"] - 1.0) / 8.0
        x = _get_neutral(tv, rv, p)
        f = torch.clamp(1.0 - x, min=TINY)
        ep = p["eta_bar"] * x / f * (bxv ** 2 + byv ** 2 + bzv ** 2) / (rv * rv) / tv.sqrt()
        B(self.eta_perp).copy_(torch.clamp(ep, max=100.0))

    # -- resistivity
    def current(self, B):
        g, bx, by, bz = self.g, self.bx, self.by, self.bz
        dx, dy, dz = (B(g.dc[d]) for d in range(3))

        def jx(o):
            a, b = tuple(np.add(o, UNIT[1])), tuple(np.add(o, UNIT[2]))
            return (B(bz, a) - B(bz, o)) / dy - (B(by, b) - B(by, o)) / dz

        def jy(o):
            a, b = tuple(np.add(o, UNIT[2])), tuple(np.add(o, UNIT[0]))
            return (B(bx, a) - B(bx, o)) / dz - (B(bz, b) - B(bz, o)) / dx

        def jz(o):
            a, b = tuple(np.add(o, UNIT[0])), tuple(np.add(o, UNIT[1]))
            return (B(by, a) - B(by, o)) / dx - (B(bx, b) - B(bx, o)) / dy
        z = (0, 0, 0)
        return (0.5 * (jx(z) + jx(UNIT[0])), 0.5 * (jy(z) + jy(UNIT[1])), 0.5 * (jz(z) + jz(UNIT[2])))

    def eta_and_fluxes(self, fluxes):
        p = self.p
        self.eta = self.zeros()
        if not p["resistive_mhd"]:
            return
        B = self.box(-1, 1)
        j = self.current(B)
        j2 = j[0] ** 2 + j[1] ** 2 + j[2] ** 2
        B(self.eta).copy_(p["eta_background"] + p["eta0"] * (j2.sqrt() > p["j_max"]).to(torch.float64))
        if not fluxes:
            return
        self.kf = [self.zeros() for _ in range(3)]
        self.curlb = self.zeros()
        B = self.box(0, 0)
        j, e = self.current(B), B(self.eta)
        if p["cowling_resistivity"]:
            bx, by, bz = self.bx, self.by, self.bz
            b = [0.25 * (B(bx) + B(bx, _off(1)) + B(bx, _off(2)) + B(bx, _off(1, 2))),
                 0.25 * (B(by) + B(by, _off(0)) + B(by, _off(2)) + B(by, _off(0, 2))),
                 0.25 * (B(bz) + B(bz, _off(0)) + B(bz, _off(1)) + B(bz, _off(0, 1)))]
            b2 = b[0] ** 2 + b[1] ** 2 + b[2] ** 2
            jb = torch.where(b2 > TINY, (j[0] * b[0] + j[1] * b[1] + j[2] * b[2]) / b2, 0.0)
            par = [jb * b[d] for d in range(3)]
            perp = [j[d] - par[d] for d in range(3)]
            ep = B(self.eta_perp)
            B(self.curlb).copy_(e * sum(q * q for q in par) + (ep + e) * sum(q * q for q in perp))
            f = [-((par[d] + perp[d]) * e + perp[d] * ep) * B(self.g.dc[d]) * 0.5 for d in range(3)]
        else:
            B(self.curlb).copy_(e * (j[0] ** 2 + j[1] ** 2 + j[2] ** 2))
            f = [-j[d] * e * B(self.g.dc[d]) * 0.5 for d in range(3)]
        for d in range(3):
            B(self.kf[d]).copy_(f[d])

    def resistive_update(self, dt):
        g = self.g
        kx, ky, kz = self.kf
        X, Y, Z, XY, XZ, YZ = _off(~0), _off(~1), _off(~2), _off(~0, ~1), _off(~0, ~2), _off(~1, ~2)
        B = self.box((0, 1, 1), 0)
        B(self.bx).add_((B(kz) - B(kz, Y) + B(kz, Z) - B(kz, YZ) - B(ky) + B(ky, Z) - B(ky, Y) + B(ky, YZ)) * dt
                        / (B(g.db[1]) * B(g.db[2])))
        B = self.box((1, 0, 1), 0)
        B(self.by).add_((B(kx) - B(kx, Z) + B(kx, X) - B(kx, XZ) - B(kz) + B(kz, X) - B(kz, Z) + B(kz, XZ)) * dt
                        / (B(g.db[0]) * B(g.db[2])))
        B = self.box((1, 1, 0), 0)
        B(self.bz).add_((B(ky) - B(ky, X) + B(ky, Y) - B(ky, XY) - B(kx) + B(kx, Y) - B(kx, X) + B(kx, XY)) * dt
                        / (B(g.db[0]) * B(g.db[1])))
        self.fill_b()
        B = self.box(1, 0)
        c = self.curlb
        B(self.energy).add_(sum(B(c, tuple(-q for q in o)) for o in CORNERS) * dt / (8.0 * B(self.rho)))
        B = self.box(-1, 2)
        B(self.energy).clamp_(min=0.0)
        B = self.box(0, 0)
        w = dt * B(g.dc[0]) * B(g.dc[1]) * B(g.dc[2]) * B(c)
        self.ohm_tot += float((w * self.half_edges()).sum())
        self.fill(self.energy, "ccc")

    def half_edges(self):
        w = 1.0
        for d in range(3):
            h = torch.ones(self.n[d] + 1, dtype=torch.float64, device=self.dev)
            h[0] = h[-1] = 0.5
            w = w * h.view([-1 if q == 2 - d else 1 for q in range(3)])
        return w

    # -- conduction
    def temperature(self, e):
        return (self.p["gamma"] - 1.0) / (2.0 - self.xi) * (e - (1.0 - self.xi) * self.p["ionise_pot"])

    def conduction_limits(self):
        """The Larsen factor over 0:n and the explicit limit."""
        p, g = self.p, self.g
        T = self.temperature(self.energy)
        B = self.box(0, 0)
        t0 = B(T)
        larsen = self.zeros()
        if p["heat_flux_limiter"]:
            qf = p["flux_limiter"] * 42.85 * B(self.rho) * t0 ** 1.5
            q2 = 0.0
            for d in range(3):
                q2 = q2 + (p["kappa_0"] * t0 ** 2.5 * (B(T, _off(d)) - B(T, _off(~d))) * 0.5 / B(g.db[d])) ** 2
            B(larsen).copy_(qf / (qf * qf + q2).sqrt())
        else:
            B(larsen).fill_(1.0)
        B = self.box(1, 0)
        h = torch.minimum(torch.minimum(B(g.db[0]) ** 2, B(g.db[1]) ** 2), B(g.db[2]) ** 2)
        lim = B(self.rho) * h / (2.0 * p["kappa_0"] * B(larsen) * B(T) ** 2.5)
        return larsen, p["dt_multiplier"] * min(float(lim.min()), 1e10) / math.sqrt(3.0)

    def stages(self, dt, limit):
        s = math.ceil(0.5 * (math.sqrt(9.0 + 16.0 * (dt / limit)) - 1.0))
        return s + 1 if s % 2 == 0 else s

    def heat_flux(self, T, larsen, coef):
        """The divergence of the limited flux over 1:n; coef: kept between stages."""
        p, g = self.p, self.g
        div = self.zeros()
        Bi = self.box(1, 0)
        rp = p["kappa_perp_ratio"]
        for d in range(3):
            e, f = [q for q in range(3) if q != d]
            lo = [1, 1, 1]
            lo[d] = 0
            B = self.box(tuple(lo), 0)
            D = UNIT[d]
            if d not in coef:
                b = (self.bx, self.by, self.bz)
                b0 = B(b[d])
                be, bf = (0.25 * (B(b[q]) + B(b[q], D) + B(b[q], _off(~q)) + B(b[q], _off(~q, d))) for q in (e, f))
                mod = b0 * b0 + be * be + bf * bf + 1.0e-10
                w = B(larsen) / mod / B(g.db[d])
                ce = B(g.dc[e]) + B(g.dc[e], _off(~e))
                cf = B(g.dc[f]) + B(g.dc[f], _off(~f))
                coef[d] = (w * (b0 * b0 + 1.0e-10 + rp * (mod - b0 * b0)) / B(g.dc[d]),
                           w * b0 * be * (1.0 - rp) * 0.5 / ce, w * b0 * bf * (1.0 - rp) * 0.5 / cf)
            kn, ke, kf = coef[d]
            tb = torch.clamp((B(T) + B(T, D)) * 0.5, min=0.0)
            grad = kn * (B(T, D) - B(T))
            for q, kq in ((e, ke), (f, kf)):
                grad = grad + kq * ((B(T, _off(q, d)) + B(T, _off(q))) - (B(T, _off(~q, d)) + B(T, _off(~q))))
            flux = self.zeros()
            B(flux).copy_(-p["kappa_0"] * tb ** 2.5 * grad)
            Bi(div).add_(Bi(flux, _off(~d)) - Bi(flux))
        return div

    def conduct(self, dt, larsen, s):
        w1 = 4.0 / (s * s + s - 2.0)
        b = [1.0 / 3.0] * 3 + [(j * j + j - 2.0) / (2.0 * j * (j + 1.0)) for j in range(3, s + 1)]
        coef = {}
        Bi = self.box(1, 0)
        y0 = self.energy
        lc0 = self.heat_flux(self.temperature(y0), larsen, coef) / torch.where(self.rho != 0, self.rho, 1.0)
        y1, y2 = y0, y0.clone()
        Bi(y2).copy_(Bi(y0) + w1 / 3.0 * dt * Bi(lc0))
        self.fill(y2, "ccc", mpi=False)
        for j in range(2, s + 1):
            mt = (2.0 * j - 1.0) / j * w1 * (b[j] / b[j - 1])
            mu = (2.0 * j - 1.0) / j * (b[j] / b[j - 1])
            nu = -(j - 1.0) / j * (b[j] / b[j - 2])
            gt = -(1.0 - b[j - 1]) * mt
            lc = self.heat_flux(self.temperature(y2), larsen, coef)
            y3 = y0.clone()
            Bi(y3).copy_(mu * Bi(y2) + nu * Bi(y1) + (1.0 - mu - nu) * Bi(y0) + mt * dt * Bi(lc) / Bi(self.rho)
                         + gt * dt * Bi(lc0))
            if j < s:
                self.fill(y3, "ccc")
            y1, y2 = y2, y3
        Bi(self.energy).copy_(Bi(y2))
        self.fill(self.energy, "ccc")

    # -- shock viscosity
    def shock_viscosity(self):
        p, g, cv = self.p, self.g, self.cv
        v = (self.vx, self.vy, self.vz)
        B = self.box(-1, 2)
        self.pressure = self.zeros()
        pr = (p["gamma"] - 1.0) * B(self.rho) * (B(self.energy) - (1.0 - (B(self.xi) if self.pip else self.xi)) * p["ionise_pot"])
        B(self.pressure).copy_(pr)
        b2 = 0.0
        for d, b in enumerate((self.bx, self.by, self.bz)):
            b2 = b2 + ((B(b) + B(b, _off(~d))) * 0.5) ** 2
        cs = self.zeros()
        B(cs).copy_(((p["gamma"] * pr + b2) / torch.clamp(B(self.rho), min=TINY)).sqrt())
        B = self.box(-1, 1)
        self.rho_v, self.cv_v, cs_v = self.zeros(), self.zeros(), self.zeros()
        csum = sum(B(cv, o) for o in CORNERS)
        B(self.rho_v).copy_(sum(B(self.rho, o) * B(cv, o) for o in CORNERS) / csum)
        B(self.cv_v).copy_(0.125 * csum)
        B(cs_v).copy_(sum(B(cs, o) * B(cv, o) for o in CORNERS) / csum)
        dt, v2n = self.dt, 0.25 * (p["gamma"] + 1.0) * p["visc2"]

        def edge(B, comp, i1, i2, dx):
            dv = [B(c, i1) - B(c, i2) for c in v]
            r1, r2 = B(self.rho_v, i1), B(self.rho_v, i2)
            re = 2.0 * r1 * r2 / (r1 + r2)
            ce = torch.minimum(B(cs_v, i1), B(cs_v, i2))
            d2 = dv[0] ** 2 + dv[1] ** 2 + dv[2] ** 2
            m = d2.sqrt()
            dd = torch.where(m * dt / dx < 1e-14, 0.0, -dv[comp].abs() / torch.where(m > 0, m, 1.0))
            return re * (v2n * m + (v2n * v2n * d2 + (p["visc1"] * ce) ** 2).sqrt()) * dd
        al = [self.zeros() for _ in range(3)]
        B = self.box(0, (1, 2, 2))
        B(al[0]).copy_(edge(B, 0, _off(~0, ~1, ~2), _off(~1, ~2), B(g.db[0])))
        B = self.box((-1, 0, 0), (1, 1, 2))
        B(al[1]).copy_(edge(B, 1, _off(~1, ~2), _off(~2), B(g.db[1])))
        B = self.box((-1, -1, 0), 1)
        B(al[2]).copy_(edge(B, 2, _off(~2), (0, 0, 0), B(g.db[2])))
        self.al = al
        # p_visc and the heating over 0:n+1, the forces over 0:n
        B = self.box(0, 1)
        self.p_visc, self.visc_heat = self.zeros(), self.zeros()
        pv = torch.zeros_like(B(self.p_visc))
        for a, i1, i2 in ((al[0], _off(~0, ~1, ~2), _off(~1, ~2)), (al[1], _off(~1, ~2), _off(~2)),
                          (al[2], _off(~2), (0, 0, 0))):
            pv = torch.maximum(pv, -B(a) * sum((B(c, i1) - B(c, i2)) ** 2 for c in v).sqrt())
        B(self.p_visc).copy_(pv)
        B(self.visc_heat).copy_(self.edge_heating(B, v, v))
        B = self.box(0, 0)
        dc = [B(g.dc[d]) for d in range(3)]
        a1, a2, a3 = al
        self.fv = []
        for c in v:
            f = (B(a1, _off(1, 2)) * dc[1] * dc[2] * (B(c) - B(c, _off(~0)))
                 + B(a1, _off(0, 1, 2)) * dc[1] * dc[2] * (B(c) - B(c, _off(0)))
                 + B(a2, _off(2)) * dc[0] * dc[2] * (B(c) - B(c, _off(~1)))
                 + B(a2, _off(1, 2)) * dc[0] * dc[2] * (B(c) - B(c, _off(1)))
                 + B(a3) * dc[0] * dc[1] * (B(c) - B(c, _off(~2)))
                 + B(a3, _off(2)) * dc[0] * dc[1] * (B(c) - B(c, _off(2)))) / B(self.cv_v)
            self.fv.append(f)

    def edge_heating(self, B, v, w):
        """The heating of a cell's twelve edges, dv . dw weighted."""
        g, (a1, a2, a3) = self.g, self.al
        dx, dy, dz = (B(g.db[d]) for d in range(3))
        heat = 0.0
        # (edge viscosity and its offset, the widths, the two corners)
        c = {"": (0, 0, 0), "x": _off(~0), "y": _off(~1), "z": _off(~2), "xy": _off(~0, ~1), "xz": _off(~0, ~2),
             "yz": _off(~1, ~2), "xyz": _off(~0, ~1, ~2)}
        edges = [(a1, (0, 0, 0), dy * dz, "xyz", "yz"), (a2, (0, 0, 0), dx * dz, "yz", "z"),
                 (a1, _off(1), dy * dz, "z", "xz"), (a2, _off(~0), dx * dz, "xz", "xyz"),
                 (a1, _off(2), dy * dz, "xy", "y"), (a2, _off(2), dx * dz, "y", ""),
                 (a1, _off(1, 2), dy * dz, "", "x"), (a2, _off(~0, 2), dx * dz, "x", "xy"),
                 (a3, (0, 0, 0), dx * dy, "z", ""), (a3, _off(~0), dx * dy, "xz", "x"),
                 (a3, _off(~0, ~1), dx * dy, "xyz", "xy"), (a3, _off(~1), dx * dy, "yz", "y")]
        for a, o, area, i, j in edges:
            dd = sum((B(p, c[i]) - B(p, c[j])) * (B(q, c[i]) - B(q, c[j])) for p, q in zip(v, w))
            heat = heat - 0.25 * area * B(a, o) * dd
        return heat / B(self.cv)

    # -- dt
    def set_dt(self):
        p, g = self.p, self.g
        B = self.box(0, 0)
        w1 = B(self.bx) ** 2 + B(self.by) ** 2 + B(self.bz) ** 2
        r = torch.clamp(B(self.rho), min=TINY)
        cs2, cq2 = (p["gamma"] * B(self.pressure) + w1) / r, B(self.p_visc) / r
        db = [B(g.db[d]) for d in range(3)]
        length = torch.minimum(torch.minimum(db[0], db[1]), db[2])
        dt = float((length / (cq2.sqrt() + (cs2 + cq2).sqrt())).min())
        for d, v in enumerate((self.vx, self.vy, self.vz)):
            dt = min(dt, float((db[d] / torch.clamp(B(v).abs(), min=TINY)).min()))
        dtr = 1.7976931348623157e308
        if p["resistive_mhd"]:
            dl = 1.0 / (1.0 / db[0] ** 2 + 1.0 / db[1] ** 2 + 1.0 / db[2] ** 2)
            e = B(self.eta)
            if p["cowling_resistivity"]:
                e = torch.maximum(e, B(self.eta_perp))
            dtr = float((0.2 * dl / torch.clamp(e, min=TINY)).min())
        self.dt, self.dtr = p["dt_multiplier"] * dt, p["dt_multiplier"] * dtr
        if p["conduction"]:
            s = self.stages(self.dt, self.conduction_limits()[1])
            if s >= 60:
                f = (2.0 * 60 * 60 - 9.0) / (2.0 * s * s - 9.0)
                self.dt, self.dtr = self.dt * f, self.dtr * f
        self.time += self.dt

    # -- remap
    def face_velocity(self, B, d, v, o=(0, 0, 0)):
        e, f = [q for q in range(3) if q != d]
        sh = lambda *a: tuple(np.add(o, _off(*a)))  # noqa: E731
        return 0.25 * (B(v, o) + B(v, sh(~e)) + B(v, sh(~f)) + B(v, sh(~e, ~f)))

    def volumes(self, a, v, dt, swept):
        """cv1, cv2 and the moved widths db1 and dc1 along axis a; swept:
        axes already done, whose terms drop out."""
        g = self.g
        B = self.box(-1, 2)
        cv1, cv2, db1, dc1 = (self.zeros() for _ in range(4))
        dv = [self.face_velocity(B, d, v[d]) - self.face_velocity(B, d, v[d], _off(~d)) for d in range(3)]
        t2 = sum(dv[d] / B(g.db[d]) for d in range(3) if d != a and d not in swept)
        B(cv1).copy_(B(self.cv) * (1.0 + (t2 + dv[a] / B(g.db[a])) * dt))
        B(cv2).copy_(B(self.cv) * (1.0 + t2 * dt) if not isinstance(t2, int) else B(self.cv).expand(B(cv2).shape))
        B(db1).copy_(B(g.db[a]) + dv[a] * dt)
        nxt = torch.cat([B(db1).narrow(2 - a, 1, self.n[a] + 3), B(db1).narrow(2 - a, self.n[a] + 3, 1)], dim=2 - a)
        B(dc1).copy_(0.5 * (B(db1) + nxt))
        return cv1, cv2, db1, dc1

    @staticmethod
    def limited(v, f, dxc, dxb, phi):
        """Van Leer's upwind value and correction from f at -1, 0, 1, 2 and
        the divisors dxc at 0, upwind."""
        up = v >= 0.0
        fm, f0, fp, f2 = f
        d0 = fp - f0
        du = torch.where(up, f0 - fm, f2 - fp)
        da = ((2.0 - phi) * d0.abs() / dxc[0] + (1.0 + phi) * du.abs() / dxc[1]) / 6.0
        same = 0.5 * (torch.copysign(torch.ones_like(d0), d0) + torch.copysign(torch.ones_like(du), du))
        sg = 2.0 * up.to(torch.float64) - 1.0
        return torch.where(up, f0, fp), sg * same * torch.minimum(torch.minimum(da.abs() * dxb, d0.abs()), du.abs())

    def sweep_b(self, a, va, dt, db1, dc1):
        """The two constrained-transport fluxes and updates (B in flux form)."""
        b = [self.bx, self.by, self.bz]
        others = [d for d in range(3) if d != a]
        A = UNIT[a]
        fl = []
        for t in others:
            o = 3 - a - t
            B = self.box(-1, 1)
            f = self.zeros()
            # B over the width at the face of component t, and its clamped neighbours
            w = self.zeros()
            lo, hi = [-1] * 3, [2] * 3
            hi[t] = 1
            W = self.box(tuple(lo), tuple(hi))
            W(w).copy_(0.5 * (W(db1) + W(db1, UNIT[t])))
            q = torch.where(w != 0, b[t] / torch.where(w != 0, w, 1.0), 0.0)
            qm, dm = self.clamped(B, q, a, -1), self.clamped(B, dc1, a, -1)
            q2 = self.clamped(B, q, a, 2)
            v = 0.5 * (B(va) + B(va, _off(~o)))
            up = v >= 0.0
            phi = v.abs() * dt / torch.where(up, B(w), B(w, A))
            fu, di = self.limited(v, (qm, B(q), B(q, A), q2), (B(dc1), torch.where(up, dm, B(dc1, A))),
                                  torch.where(up, B(db1), B(db1, A)), phi)
            B(f).copy_((fu + di * (1.0 - phi)) * v * dt)
            fl.append((t, f))
        Bu = self.box(0, 1)
        back = _off(~a)
        (t1, f1), (t2, f2) = fl
        Bu(b[t1]).add_(Bu(f1, back) - Bu(f1))
        Bu(b[a]).add_(Bu(f1) - Bu(f1, _off(~t1)))
        # the second flux's own ranges, file by file
        lo, hi, lob, hib = [0] * 3, [1] * 3, [0] * 3, [1] * 3
        if a == 0:
            lo, hi = [1, 1, 0], [0, 0, 0]
            hib = [0, 1, 1]
        elif a == 1:
            lob, hib = [1, 0, 1], [0, 0, 0]
        Bu = self.box(tuple(lo), tuple(hi))
        Bu(b[t2]).add_(Bu(f2, back) - Bu(f2))
        Bu = self.box(tuple(lob), tuple(hib))
        Bu(b[a]).add_(Bu(f2) - Bu(f2, _off(~t2)))

    def clamped(self, B, x, a, off):
        """x at index + off along a, the index held inside -1..n+2."""
        n, lo, hi = self.n[a], B.lo[a], B.hi[a]
        idx = torch.arange(lo, hi + 1, device=self.dev)
        idx = torch.clamp(idx + off, -1, n + 2) + 2
        wide = list(B.lo), list(B.hi)
        wide[0][a], wide[1][a] = -2, n + 2
        return _Box(*wide)(x).index_select(2 - a, idx)

    def flux_form(self, inverse):
        g = self.g
        for d, name in enumerate(("bx", "by", "bz")):
            area = g.db[(d + 1) % 3] * g.db[(d + 2) % 3]
            b = getattr(self, name)
            setattr(self, name, b / area if inverse else b * area)

    def remap_b(self, v, dt, step):
        self.flux_form(False)
        for a in ORDER[step % 6]:
            cv1, _cv2, db1, dc1 = self.volumes(a, v, dt, ())
            self.sweep_b(a, v[a], dt, db1, dc1)
        self.flux_form(True)
        self.fill_b()
        return cv1

    def sweep(self, a, v1, dt, swept):
        g = self.g
        cv1, cv2, db1, dc1 = self.volumes(a, v1, dt, swept)
        self.sweep_b(a, v1[a], dt, db1, dc1)
        t1, t2 = [d for d in range(3) if d != a]
        n, A, A2 = self.n, UNIT[a], tuple(2 * q for q in UNIT[a])
        back = _off(~a)
        # mass flux
        lo, hi = [0] * 3, [1] * 3
        lo[a], hi[a] = (1 if self.per[a] else 0), 0
        B = self.box(tuple(lo), tuple(hi))
        area = g.db[t1] * g.db[t2]

        def scalar(B, f, other):
            v = self.face_velocity(B, a, v1[a])
            up = v >= 0.0
            dxb = torch.where(up, B(db1), B(db1, A))
            phi = v.abs() * dt / dxb
            fu, di = self.limited(v, (B(f, back), B(f), B(f, A), B(f, A2)),
                                  (B(dc1), torch.where(up, B(dc1, back), B(dc1, A))), dxb, phi)
            return v, up, dxb, phi, fu, di
        v, up, dxb, phi, fu, di = scalar(B, self.rho, None)
        dm = self.zeros()
        B(dm).copy_((fu + di * (1.0 - phi)) * v * dt * B(area))
        d = dm.movedim(2 - a, 0)
        if self.per[a]:
            for i, j in ((n[a] + 1, 1), (n[a] + 2, 2), (-1, n[a] - 1), (0, n[a])):
                d[i + 2] = d[j + 2]
        else:
            d[n[a] + 3] = d[n[a] + 2]
            d[1] = d[2]
        # density and energy
        rho1 = self.rho
        rho = rho1.clone()
        B = self.box(1, 0)
        B(rho).copy_((B(rho1) * B(cv1) + B(dm, back) - B(dm)) / B(cv2))
        ef = self.zeros()
        B0 = self.box(0, 0)
        v, up, dxb, phi, fu, di = scalar(B0, self.energy, None)
        rhou = torch.where(up, B0(rho1), B0(rho1, A))
        dmu = B0(dm).abs() / B0(area) / dxb / rhou
        B0(ef).copy_((fu + di * (1.0 - dmu)) * B0(dm))
        B(self.energy).copy_((B(self.energy) * B(cv1) * B(rho1) + B(ef, back) - B(ef)) / (B(cv2) * B(rho)))
        # vertex averages
        rv, rv1, cv1v, cv2v, dmv = (self.zeros() for _ in range(5))
        lo, hi = [0] * 3, [0] * 3
        lo[a], hi[a] = -1, 1
        V = self.box(tuple(lo), tuple(hi))
        V(cv1v).copy_(0.125 * sum(V(cv1, o) for o in CORNERS))
        V(rv).copy_(sum(V(rho1, o) * V(cv1, o) for o in CORNERS) / (8.0 * V(cv1v)))
        hi[a] = 0
        V = self.box(tuple(lo), tuple(hi))
        V(dmv).copy_(0.125 * sum(V(dm, o) for o in CORNERS))
        U = self.box(0, 0)
        U(cv2v).copy_(0.125 * sum(U(cv2, o) for o in CORNERS))
        U(rv1).copy_((U(rv) * U(cv1v) + U(dmv, back) - U(dmv)) / U(cv2v))
        # momentum: faces -1:n along a
        F = V
        va = 0.5 * (F(v1[a]) + F(v1[a], A))
        up = va >= 0.0
        dxb = torch.where(up, F(dc1), F(dc1, A))
        phi = va.abs() * dt / dxb
        rhou = torch.where(up, F(rv), F(rv, A))
        dmu = F(dmv).abs() / (F(g.dc[t1]) * F(g.dc[t2])) / dxb / rhou
        new = []
        for c in (self.vx, self.vy, self.vz):
            fu, di = self.limited(va, (F(c, back), F(c), F(c, A), F(c, A2)),
                                  (F(db1, A), torch.where(up, F(db1), F(db1, A2))), dxb, phi)
            fl = self.zeros()
            F(fl).copy_((fu + di * (1.0 - dmu)) * F(dmv))
            u = self.zeros()
            U(u).copy_((U(rv) * U(c) * U(cv1v) + U(fl, back) - U(fl)) / (U(cv2v) * U(rv1)))
            new.append(u)
        self.vx, self.vy, self.vz = new
        self.rho = rho
        self.boundary_conditions()

    # -- the step
    def step(self, step):
        p, g = self.p, self.g
        if self.pip:
            self.xi = self.neutral_fraction(self.energy)
        self.shock_viscosity()
        self.set_dt()
        if p["resistive_mhd"]:
            sub = int(self.dt / self.dtr) + 1
            for _ in range(sub):
                if self.pip:
                    self.xi = self.neutral_fraction(self.energy)
                if p["cowling_resistivity"]:
                    self.perpendicular_resistivity()
                self.eta_and_fluxes(True)
                self.resistive_update(self.dt / sub)
        if p["conduction"]:
            larsen, limit = self.conduction_limits()
            self.conduct(self.dt, larsen, self.stages(self.dt, limit))
        dt, dt2 = self.dt, 0.5 * self.dt
        v = [self.vx, self.vy, self.vz]
        # predictor: B at the half step, the half-step velocity
        b0 = (self.bx, self.by, self.bz)
        cv1 = self.remap_b(v, dt2, step)
        B = self.box(-1, 2)
        B(self.energy).clamp_(min=0.0)
        B = self.box(0, 1)
        rho = B(self.rho)
        e1 = B(self.energy) - B(self.pressure) * (B(cv1) / B(self.cv) - 1.0) / rho + B(self.visc_heat) * dt2 / rho
        xi = B(self.xi) if self.pip else self.xi
        B(self.pressure).copy_((e1 - (1.0 - xi) * p["ionise_pot"]) * (p["gamma"] - 1.0) * rho * B(self.cv) / B(cv1))
        B = self.box(0, 0)
        f = []
        for d in range(3):
            e, h = [q for q in range(3) if q != d]
            lo = [(0, 0, 0), _off(e), _off(h), _off(e, h)]
            near = sum(B(self.pressure, o) for o in lo) * 0.25
            far = sum(B(self.pressure, tuple(np.add(o, UNIT[d]))) for o in lo) * 0.25
            f.append(-(far - near) / B(g.dc[d]))
        j = self.current(B)
        bv = [0.25 * (B(b) + B(b, _off(e)) + B(b, _off(h)) + B(b, _off(e, h)))
              for b, e, h in ((self.bx, 1, 2), (self.by, 0, 2), (self.bz, 0, 1))]
        f[0] = f[0] + (j[1] * bv[2] - j[2] * bv[1])
        f[1] = f[1] + (j[2] * bv[0] - j[0] * bv[2])
        f[2] = f[2] + (j[0] * bv[1] - j[1] * bv[0]) - B(self.rho_v) * B(self.grav)
        v1 = [self.zeros() for _ in range(3)]
        for d in range(3):
            B(v1[d]).copy_(B(v[d]) + dt2 * (self.fv[d] + f[d]) / B(self.rho_v))
        self.bx, self.by, self.bz = b0
        self.fill_v(v1)
        # corrector
        C = self.box(0, 1)
        heat = torch.clamp(self.edge_heating(C, v, v1), min=0.0)
        C(self.visc_heat).copy_(heat)
        for d in range(3):
            B(v[d]).copy_(2.0 * B(v1[d]) - B(v[d]))
        self.fill_v(v)
        B = self.box(1, 0)
        dv = sum((self.face_velocity(B, d, v1[d]) - self.face_velocity(B, d, v1[d], _off(~d))) / B(g.db[d])
                 for d in range(3)) * dt
        vh = B(self.visc_heat)
        B(self.energy).add_((dt * vh - dv * B(self.pressure)) / B(self.rho))
        B(self.rho).div_(1.0 + dv)
        self.visc_tot += float((dt * vh * B(self.cv)).sum())
        self.fill(self.energy, "ccc")
        self.fill(self.rho, "ccc")
        # remap
        self.flux_form(False)
        swept = []
        for a in ORDER[step % 6]:
            self.sweep(a, v1, dt, tuple(swept))
            swept.append(a)
        self.flux_form(True)
        self.fill_b()
        self.eta_and_fluxes(False)

    def account(self):
        g, cv = self.g, self.cv
        B = self.box(1, 0)
        w = 0.0
        for d, b in enumerate((self.bx, self.by, self.bz)):
            w = w + (B(b) ** 2 + B(b, _off(~d)) ** 2) * 0.5
        en_b = float((0.5 * w * B(cv)).sum())
        en_i = float((B(self.energy) * B(self.rho) * B(cv)).sum())
        B = self.box(0, 0)
        rv = 0.125 * sum(B(self.rho, o) * B(cv, o) for o in CORNERS)
        k = 0.5 * rv * (B(self.vx) ** 2 + B(self.vy) ** 2 + B(self.vz) ** 2)
        return np.array([en_b, float((k * self.half_edges()).sum()), en_i, self.visc_tot, self.ohm_tot])

    def fields(self):
        return {k: _bounded(getattr(self, k), *abi.bounds(abi.STATE_KINDS[k], *self.n)) for k in STATE}


ORDER = ((0, 1, 2), (1, 2, 0), (2, 0, 1), (0, 2, 1), (2, 1, 0), (1, 0, 2))


def _get_neutral(t, rho, p):
    """The ionisation balance (a Saha-like law with a diluted photospheric field)."""
    b = 1.0 / (0.5 * p["f_bar"] * p["tr"] * t.sqrt()) * torch.exp((0.25 * (t / p["tr"] - 1.0) + 1.0) * p["t_bar"] / t)
    r = 0.5 * (-1.0 + (1.0 + p["r_bar"] * rho * b).sqrt())
    return r / (1.0 + r)


def _conduct_dt(x):
    """Fifty explicit limits of the state."""
    return 50.0 * x.conduction_limits()[1]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "forward"):
        return _exact_network(case, seed)
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    g, p, s, dt, grav = _inputs(case, seed)
    x = _Exact(g, p, s, dt, grav)
    if kind == "conduct":
        dt = _conduct_dt(x)
        larsen, limit = x.conduction_limits()
        k = x.stages(dt, limit)
        x.conduct(dt, larsen, k)
        return dict(energy=x.fields()["energy"], stages=k)
    x.step(1)
    out = dict(time=x.time, dt=x.dt, **x.fields())
    if kind == "hosted":
        return {k: (v if isinstance(v, float) else v.permute(2, 1, 0)) for k, v in out.items()}
    return dict(account=x.account(), **out)


def _exact_ensemble(case, seed):
    """One eager step and the six of the launch, member by member."""
    got = {k: [] for k in STATE}
    for spec in _members(case, seed):
        g, p, s = _member(spec)
        x = _Exact(g, p, s, 0.0, None)
        for step in range(1, 8):
            x.step(step)
        for k, v in x.fields().items():
            got[k].append(v.reshape(-1))
    return {k: torch.cat(v) for k, v in got.items()}

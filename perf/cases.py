"""The work that users of this framework have it do, as cases that can be timed and
checked: whole DTs of single disks (isothermal, adiabatic with cooling, self-gravitating,
the reference's largest setup) in both precision modes, ensembles of disks, and the
learned correction's network.

A case is a dict of plain values; prepare() builds what a program holds before the call,
run() is one call, exact() the same result in 64-bit torch without this package.
"""
import ctypes
import math

import numpy as np
import torch

DT = 0.314159265359  # the configurations' DT: a twentieth of the orbit at r = 1


def listed():
    return [
        # one DT of the 128 x 384 isothermal disk, the smallest single-disk setup of the configurations:
        # launches and latency count
        dict(name="c1_fp64", kind="disk", config="c1", fp64=True, nrad=128, nsec=384),
        dict(name="c1_fp32", kind="disk", config="c1", fp64=False, nrad=128, nsec=384),
        # a grid whose ring is no multiple of anything: adiabatic, with cooling
        dict(name="ragged_fp64", kind="disk", config="c3", fp64=True, nrad=201, nsec=603),
        # the self-gravitating disk with a migrating planet
        dict(name="c2_fp64", kind="disk", config="c2", fp64=True, nrad=256, nsec=768),
        dict(name="c2_fp32", kind="disk", config="c2", fp64=False, nrad=256, nsec=768),
        # the large adiabatic disk with cooling: the benchmark's headline
        dict(name="c3_fp64", kind="disk", config="c3", fp64=True, nrad=1024, nsec=3072),
        dict(name="c3_fp32", kind="disk", config="c3", fp64=False, nrad=1024, nsec=3072),
        # the reference's largest setup: non-reflecting boundary, guiding-centre frame
        dict(name="wide_fp32", kind="disk", config="wide", fp64=False, nrad=2048, nsec=4096),
        # the seeded ensemble of uneven isothermal disks: one DT of every disk, per-disk graphs
        dict(name="ensemble_fp32", kind="ensemble", disks=32, least=128, most=512, fused=False),
        # many small disks, in the fused form
        dict(name="small_fused_fp32", kind="ensemble", disks=64, least=32, most=64, fused=True),
        # the correction network on every cell of a 256 x 768 disk: inference, and a training step on a ragged batch
        dict(name="mlp_forward", kind="mlp", rows=196608, train=False),
        dict(name="mlp_train", kind="mlp", rows=100003, train=True),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["disk", "disk", "disk", "disk", "ensemble", "mlp"])
    if kind == "mlp":
        return dict(kind=kind, rows=_log(rng, 100, 196608), train=rng.random() < 0.5)
    if kind == "ensemble":
        least = rng.choice([32, 64, 128])
        return dict(kind=kind, disks=_log(rng, 4, 32), least=least, most=least * rng.choice([2, 4]), fused=rng.random() < 0.5)
    config = rng.choice(["c1", "c2", "c3", "c3"])
    fp64 = rng.random() < 0.5
    if config == "c2":  # the transforms take lengths of factors 2 and 3
        nrad, nsec = rng.choice([48, 64, 96, 128, 192, 256, 384]), rng.choice([192, 256, 384, 512, 576, 768, 1024])
    else:
        nrad = _log(rng, 40, 1024)
        nsec = int(nrad * rng.uniform(2.0, 3.0))
        if rng.random() < 0.5:
            nsec = max(4, nsec // 4 * 4)
    return dict(kind=kind, config=config, fp64=fp64, nrad=nrad, nsec=nsec)


# ---- the disks' parameters, as the .par and .cfg files of the configurations have them ---------------------------

COMMON = dict(aspectratio=0.05, viscosity=0.0, alphaviscosity=0.0, self_gravity=0, adiabatic=0, cooling=0, rmin=0.4, rmax=2.5,
              adiabaticindex=1.4, coolingtime0=6.28, forced_circular=1, thicknesssmoothing=0.6, non_reflecting=0, corotating=0,
              sigma0=6.3662e-4, sigmaslope=0.5)
PHYSICS = {
    "c1": dict(COMMON, viscosity=1e-5),
    "c2": dict(COMMON, sigma0=8.84194128288308e-4, sigmaslope=1.0, alphaviscosity=1e-3, self_gravity=1, rmax=4.0, forced_circular=0,
               thicknesssmoothing=0.3),
    "c3": dict(COMMON, alphaviscosity=1e-3, adiabatic=1, cooling=1, coolingtime0=10.0, rmin=0.3, rmax=3.0),
    "wide": dict(COMMON, sigma0=5.1e-5, viscosity=1e-5, adiabatic=1, non_reflecting=1, corotating=1, forced_circular=0),
}
PLANET = {"c1": (1.0, 1e-3, False), "c2": (1.5, 5e-4, True), "c3": (1.0, 1e-3, False), "wide": (1.0, 1e-3, False)}


def _members(case, seed):
    """The disks of a case: (physics with its grid, planet distance, mass, feels the disk, seed of the fields)."""
    if case["kind"] == "disk":
        c = case["config"]
        return [(dict(PHYSICS[c], nrad=case["nrad"], nsec=case["nsec"]), *PLANET[c], seed)]
    choices = [n for n in (32, 48, 64, 96, 128, 192, 256, 384, 512) if case["least"] <= n <= case["most"]]
    sizes = np.random.Generator(np.random.PCG64(2024)).choice(choices, case["disks"])  # the case's own, whatever the seed
    rng = np.random.Generator(np.random.PCG64(seed))
    got = []
    for k, nrad in enumerate(sizes.tolist()):
        q, alpha = 10 ** rng.uniform(-5, math.log10(3e-3)), 10 ** rng.uniform(-4, -2)
        p = dict(COMMON, nrad=nrad, nsec=3 * nrad, alphaviscosity=float(alpha), aspectratio=float(rng.uniform(0.03, 0.08)),
                 sigmaslope=float(rng.uniform(0, 1.5)))
        got.append((p, 1.0, float(q), False, seed * 1000 + k))
    return got


def _mesh(p, dev="cpu"):
    """Rinf (nrad + 1), Rmed (nrad) of the logarithmic grid."""
    span = math.log(p["rmax"] / p["rmin"])
    r = torch.tensor([p["rmin"] * math.exp(k / p["nrad"] * span) for k in range(p["nrad"] + 1)], dtype=torch.float64, device=dev)
    return r, 2 / 3 * (r[1:] ** 3 - r[:-1] ** 3) / (r[1:] ** 2 - r[:-1] ** 2)


def _fields(p, seed, fp64):
    """A disk that has run for a while: the power laws with a two-armed wave and noise; zeros on ring nrad, the ghost ring."""
    nr, ns, h = p["nrad"], p["nsec"], p["aspectratio"]
    g = torch.Generator().manual_seed(seed)
    rinf, r = _mesh(p)
    r, ri = r[:, None], rinf[:-1, None]
    phi = torch.arange(ns, dtype=torch.float64)[None, :] * (2 * math.pi / ns)
    phase = float(torch.rand(1, generator=g, dtype=torch.float64)) * 2 * math.pi

    def wave(x):
        return torch.cos(2 * phi - 4 * torch.log(x) / 0.5 + phase)

    def noise(a):
        return a * (2 * torch.rand((nr, ns), generator=g, dtype=torch.float64) - 1)

    dens = p["sigma0"] * r ** -p["sigmaslope"] * (1 + 0.05 * wave(r) + noise(1e-3))
    kep = r ** -0.5 * math.sqrt(1 - h * h * (1 + p["sigmaslope"]))
    if p["corotating"]:  # rotating with the planet at r = 1
        kep = kep - r * math.sqrt(1 + 1e-3)
    vtheta = kep + 0.05 * h * r ** -0.5 * (wave(r) + noise(1e-3))
    vrad = 0.05 * h * ri ** -0.5 * (wave(ri) + noise(1e-3))
    vrad[0] = 0.0
    out = dict(dens=dens, vrad=vrad, vtheta=vtheta)
    if p["adiabatic"]:
        out["energy"] = p["sigma0"] * h * h / (p["adiabaticindex"] - 1) * r ** (-p["sigmaslope"] - 1) * (1 + 0.05 * wave(r) + noise(1e-3))
    out = {k: torch.nn.functional.pad(v, (0, 0, 0, 1)) for k, v in out.items()}
    return out if fp64 else {k: v.float().double() for k, v in out.items()}  # what a single-precision disk can hold


# ---- prepare and run ---------------------------------------------------------------------------------------------


def _mlp_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn((case["rows"], 128), generator=g)
    x[:, 125:] = 0  # the padding of the 125 inputs
    return x.bfloat16(), torch.randn((case["rows"], 2), generator=g) / case["rows"]


def _mlp_params(seed):
    """He-style weights W1 128 x 64, W2 64 x 64, W3 64 x 8 (two columns used) and biases, as the library's FP32 blob."""
    rng = np.random.default_rng(seed)
    w3, b3 = np.zeros((64, 8)), np.zeros(8)
    w3[:, :2], b3[:2] = rng.normal(0, 0.1, (64, 2)), rng.normal(0, 0.1, 2)
    parts = [rng.normal(0, 0.125, (128, 64)), rng.normal(0, 0.1, 64), rng.normal(0, 0.18, (64, 64)), rng.normal(0, 0.1, 64), w3, b3]
    return np.concatenate([v.ravel() for v in parts]).astype(np.float32)


def _params(p, dist, mass, feels):
    """FargoParams and planets of a disk, from the configuration that has its kind."""
    import cudaprotoplanetarydisks_gb300 as fg
    base = "c2" if p["self_gravity"] else "wide" if p["corotating"] else "c3" if p["adiabatic"] else "c1"
    params, planets = fg.load_config(base, sigma_noise=0.0, energy_noise=0.0, **{k: v for k, v in p.items() if k not in ("corotating", "non_reflecting")})
    if mass != planets[0].mass:
        fg.config.set_planet_mass(params, planets[0], mass)
    return params, planets


def prepare(case, seed):
    import cudaprotoplanetarydisks_gb300 as fg
    if case["kind"] == "mlp":
        from cudaprotoplanetarydisks_gb300 import learned
        x, dy = _mlp_inputs(case, seed)
        return dict(case=case, mlp=learned.MLP(case["rows"], params=_mlp_params(seed)), x=x.cuda(), dy=dy.cuda(),
                    y=torch.empty((case["rows"], 2), device="cuda"))
    fp64 = case.get("fp64", False)
    precision = fg.FARGO_FP64 if fp64 else fg.FARGO_FP32_BULK
    members = _members(case, seed)
    made = [_params(p, dist, mass, feels) for p, dist, mass, feels, _ in members]
    state = dict(case=case, fp64=fp64)
    if case["kind"] == "ensemble":
        state["batch"] = fg.Batch(made, precision)
        if case["fused"]:
            state["batch"].fuse()
        disks = state["batch"].disks
    else:
        disks = [fg.Disk(*made[0], precision)]
    for d, (p, _, _, _, s) in zip(disks, members):
        d.set_fields(**{k: v.numpy() for k, v in _fields(p, s, fp64).items()})
    names = ["dens", "vrad", "vtheta"] + (["energy"] if members[0][0]["adiabatic"] else []) + (["temperature"] if case["kind"] == "disk" else [])
    state["disks"] = disks
    # the program's own arrays of the fields, in the library's FP64 layout: one per field, the disks one after another
    cells = [(d.nrad + 1) * d.nsec for d in disks]
    state["out"] = {k: torch.zeros(sum(cells), dtype=torch.float64, device="cuda") for k in names}
    state["at"] = np.concatenate([[0], np.cumsum(cells)])
    return state


def run(state):
    import cudaprotoplanetarydisks_gb300 as fg
    if state["case"]["kind"] == "mlp":
        m = state["mlp"]
        m.forward(state["x"], state["y"])
        if not state["case"]["train"]:
            return state["y"]
        m.backward(state["x"], state["dy"])
        m.adam(1e-3)
        return dict(y=state["y"], grad=m.grad(), params=m.params())
    got = {}
    if "batch" in state:
        state["batch"].run_async(1)
        state["batch"].sync()
    else:
        got["substeps"] = state["disks"][0].step_DT()
    for name, buf in state["out"].items():
        for d, at in zip(state["disks"], state["at"]):
            rc = d.lib.fargo_get_field_device(d.h, fg.FIELDS[name], ctypes.c_void_p(buf.data_ptr() + 8 * int(at)))
            if rc:
                raise RuntimeError("get_field_device: status %d" % rc)
        # the rings that the dumps hold, without a single disk's ghost ring; FP32 fields come widened: float() gives them back as they are
        end = buf.numel() if "batch" in state else state["disks"][0].nrad * state["disks"][0].nsec
        got[name] = buf[:end] if state["fp64"] else buf[:end].float()
    return got


def work(case):
    if case["kind"] == "mlp":
        n, layer = case["rows"], 128 * 64 + 64 * 64 + 64 * 2
        params = 128 * 64 + 64 + 64 * 64 + 64 + 64 * 8 + 8
        return dict(bytes=n * (256 + 8) + 4 * params + case["train"] * (n * 8 + 6 * 4 * params), flops=2 * n * layer * (3 if case["train"] else 1))
    total = dict(bytes=0, flops=0)
    for p, *_ in _members(case, 1):
        r, rm = (v.numpy() for v in _mesh(p))
        cs = p["aspectratio"] * rm ** -0.5 * (math.sqrt(p["adiabaticindex"]) if p["adiabatic"] else 1)
        cfl = 0.5 * np.min(np.minimum(np.diff(r), rm * 2 * math.pi / p["nsec"])[1:] / cs[1:])
        shear = math.pi / p["nsec"] / np.max(-np.diff(rm ** -1.5))
        steps = math.ceil(DT / min(cfl, shear))  # the state has to be complete before the next step's length is known
        cells, fields = p["nrad"] * p["nsec"], 4 if p["adiabatic"] else 3
        e = 8 if case.get("fp64") else 4
        total["bytes"] += steps * cells * 2 * fields * e
        total["flops"] += steps * cells * (400 if p["adiabatic"] else 300)
        if p["self_gravity"]:
            total["flops"] += steps * 4 * 5 * 2 * cells * math.log2(2 * cells)
    return total


# ---- the same in 64 bits, without the package ---------------------------------------------------------------------


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed, dev)
    got = {}
    for p, dist, mass, feels, s in _members(case, seed):
        d = _Hydro(p, dist, mass, feels, {k: v.to(dev) for k, v in _fields(p, s, case.get("fp64", False)).items()}, dev)
        steps = d.dt()
        for name in ("dens", "vrad", "vtheta") + (("energy",) if p["adiabatic"] else ()) + (("temperature",) if case["kind"] == "disk" else ()):
            v = getattr(d, name)
            got.setdefault(name, []).append((v[:-1] if case["kind"] == "disk" else v).reshape(-1).cpu())
    out = {k: torch.cat(v) for k, v in got.items()}
    if case["kind"] == "disk":
        out["substeps"] = steps
    return out


def _exact_mlp(case, seed, dev):
    x, dy = _mlp_inputs(case, seed)
    x, dy = x.to(dev).double(), dy.to(dev).double()
    blob = torch.from_numpy(_mlp_params(seed)).to(dev).double().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(blob, [128 * 64, 64, 64 * 64, 64, 64 * 8, 8])

    def gelu(z):
        return torch.nn.functional.gelu(z, approximate="tanh")

    h = gelu(gelu(x @ w1.view(128, 64) + b1) @ w2.view(64, 64) + b2)
    y = h @ w3.view(64, 8)[:, :2] + b3[:2]
    if not case["train"]:
        return y.detach().cpu()
    (y * dy).sum().backward()
    g = blob.grad
    after = blob.detach() - 1e-3 * g / (g.abs() + 1e-8)  # Adam's first step, its moments' bias corrected
    return dict(y=y.detach().cpu(), grad=g.cpu(), params=after.cpu())


class _Hydro:
    """One disk of the FARGO-ADSG scheme in 64 bits, whole fields at a time: a DT as the reference's AlgoGas takes it."""

    def __init__(self, p, dist, mass, feels, f, dev):
        self.p, self.dev, self.nr, self.ns = p, dev, p["nrad"], p["nsec"]
        nr, ns, h, g = self.nr, self.ns, p["aspectratio"], p["adiabaticindex"]
        r, rm = _mesh(p, dev)
        self.r, self.rm = r[:, None], rm[:, None]  # interfaces 0..nrad, centres 0..nrad-1
        self.ri, self.rs = self.r[:-1], self.r[1:]
        self.surf = math.pi * (self.rs ** 2 - self.ri ** 2) / ns
        self.drm = self.rm[1:] - self.rm[:-1]
        self.dphi = 2 * math.pi / ns
        self.dx = self.rm * self.dphi
        a = torch.arange(ns, dtype=torch.float64, device=dev) * self.dphi
        self.x, self.y = self.rm * torch.cos(a), self.rm * torch.sin(a)
        self.dens, self.vrad, self.vtheta = f["dens"], f["vrad"], f["vtheta"]
        self.energy = f.get("energy")
        self.temperature = torch.zeros_like(self.dens)
        self.smed = p["sigma0"] * self.rm ** -p["sigmaslope"]
        self.emed = h * h * p["sigma0"] / (g - 1) * self.rm ** (-p["sigmaslope"] - 1)
        self.cs = (h * self.rm ** -0.5).expand(nr, ns)
        v0 = math.sqrt((1 + mass) / dist)
        self.m, self.feels, self.pl = mass, feels, [dist, 0.0, -1e-10 * v0, v0]
        self.om, self.t = 0.0, 0.0
        if p["adiabatic"]:  # the initial disk's sound speed: it sets the cooling's reference heating
            c0 = torch.sqrt(g * (g - 1) * self.emed / self.smed)
        else:
            c0 = h * self.rm ** -0.5
        nu0 = self._nu(c0)
        self.qmed = 2.25 * nu0 * p["sigma0"] * self.rm ** (-p["sigmaslope"] - 3)
        self.tcool = p["coolingtime0"] * self.rm ** 2
        self.vkep2 = 1 / self.rm * (1 - (1 + p["sigmaslope"]) * h * h)
        if p["self_gravity"]:
            self._gravity_kernels()
            axi, _ = self._gravity((self.smed + torch.zeros_like(self.x)))
            axi = axi.mean(1).cpu()
            c = rm.cpu()
            k = min(int((c <= dist).sum()), nr - 2)
            acc = float(((dist - c[k]) * axi[k + 1] + (c[k + 1] - dist) * axi[k]) / (c[k + 1] - c[k]))
            self.pl[3] *= math.sqrt(1 - dist * dist * acc)
        if p["corotating"]:
            self.om = self._orbit()[0]

    def _nu(self, cs):
        p = self.p
        return p["alphaviscosity"] * cs.mean(1, keepdim=True) ** 2 * self.rm ** 1.5 if p["alphaviscosity"] else torch.full_like(self.rm, p["viscosity"])

    # the planet

    def _orbit(self):
        """Angular frequency and guiding centre of the planet's osculating orbit."""
        x, y, vx, vy = self.pl
        m = 1 + self.m
        h, d = x * vy - y * vx, math.hypot(x, y)
        ax, ay = x * vy * vy - y * vx * vy - m * x / d, y * vx * vx - x * vx * vy - m * y / d
        e = math.hypot(ax, ay) / m
        a = h * h / m / (1 - e * e)
        arg = 1.0 if e == 0 else (1 - d / a) / e
        E = math.pi * (1 - arg / abs(arg)) / 2 if abs(arg) >= 1 else math.acos(arg)
        if x * y * (vy * vy - vx * vx) + vx * vy * (x * x - y * y) < 0:
            E = -E
        M, pa = E - e * math.sin(E), math.atan2(ay, ax)
        c = (x, y) if e < 1e-8 else (a * math.cos(M + pa), a * math.sin(M + pa))
        return math.sqrt(m / a ** 3), c

    def _kepler(self, q, dt):
        """One step of the fifth-order Runge-Kutta scheme (Cash and Karp's coefficients)."""
        def deriv(s):
            d3 = math.hypot(s[0], s[1]) ** 3
            k = -(1 + self.m) / d3
            return [dt * s[2], dt * s[3], dt * k * s[0], dt * k * s[1]]

        rows = [[], [0.2], [0.075, 0.225], [0.3, -0.9, 1.2], [-11 / 54, 2.5, -70 / 27, 35 / 27],
                [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
        ks = []
        for row in rows:
            ks.append(deriv([q[i] + sum(c * k[i] for c, k in zip(row, ks)) for i in range(4)]))
        w = [37 / 378, 0, 250 / 621, 125 / 594, 0, 512 / 1771]
        return [q[i] + sum(c * k[i] for c, k in zip(w, ks)) for i in range(4)]

    def _advance_planet(self, dt):
        x, y, vx, vy = self.pl
        if not self.p["forced_circular"]:
            self.pl = self._kepler(self.pl, dt)
            return
        th, r = math.atan2(y, x), math.hypot(x, y)
        d = (x * vy - y * vx) / r / r * dt
        self.pl = [r * math.cos(th + d), r * math.sin(th + d), vx * math.cos(d + th) - vy * math.sin(d + th), vx * math.sin(d + th) + vy * math.cos(d + th)]

    def _pull(self, x, y, eps):
        dx, dy = self.x - x, self.y - y
        d2 = dx * dx + dy * dy + eps * eps
        w = self.surf * self.dens[:-1] / d2 / torch.sqrt(d2)
        return float((w * dx).sum()), float((w * dy).sum())

    # self-gravity: the convolution in log r and azimuth, padded to twice the rings

    def _gravity_kernels(self):
        p, nr, dev = self.p, self.nr, self.dev
        self.eps, self.rstep = p["thicknesssmoothing"] * p["aspectratio"], math.log(p["rmax"] / p["rmin"]) / nr
        u = torch.tensor([math.log(v / p["rmin"]) for v in self.r[:, 0].tolist()], dtype=torch.float64, device=dev)
        u = torch.cat([u[:-1], -torch.flip(u[1:], [0])])[:, None]
        th = (torch.arange(self.ns, dtype=torch.float64, device=dev) * self.dphi)[None]
        coshf = ctypes.CDLL("libm.so.6").coshf  # the scheme takes it in single precision, from the C library
        coshf.restype, coshf.argtypes = ctypes.c_float, [ctypes.c_float]
        cosh = torch.tensor([coshf(v) for v in u[:, 0].tolist()], dtype=torch.float64, device=dev)[:, None]
        base = (self.eps ** 2 * torch.exp(u) + 2 * (cosh - torch.cos(th))) ** -1.5
        self.kr = torch.fft.fft2((1 + self.eps ** 2 - torch.cos(th) * torch.exp(-u)) * base)
        self.kt = torch.fft.fft2(torch.sin(th) * base)

    def _gravity(self, dens):
        q = self.rm / self.rm[0]

        def conv(s, k):
            s = torch.nn.functional.pad(s, (0, 0, 0, self.nr))
            return -torch.fft.ifft2(torch.fft.fft2(s) * k).real[:self.nr] * self.rstep * self.dphi

        ar = conv(dens * q.sqrt(), self.kr) / q.sqrt() + dens * self.rstep * self.dphi / self.eps
        return ar, conv(dens * q ** 1.5, self.kt) / q ** 1.5

    # the gas

    def _limit(self, left):
        """The number of equal steps that the time left is cut into (ConditionCFL)."""
        vr, vt = self.vrad, self.vtheta[:-1]
        mean = vt.mean(1, keepdim=True)
        dr = self.rs - self.ri
        a = self.cs / torch.minimum(dr, self.dx)
        b, c = vr[:-1].abs() / dr, (vt - mean).abs() / self.dx

        def shrink(d):
            return torch.where(d >= 0, torch.full_like(d, 1e-10), -d)

        e = 4 * 1.41 * 1.41 * torch.maximum(shrink(vr[1:] - vr[:-1]) / dr, shrink(torch.roll(vt, -1, 1) - vt) / self.dx)
        cell = 0.5 / math.sqrt(float((a * a + b * b + c * c + e * e)[1:].max()))
        w = mean / self.rm
        shear = math.pi / self.ns / float((w[1:] - w[:-1]).abs().max())
        return math.ceil(left / min(cell, shear, left))

    def dt(self):
        p, g = self.p, self.p["adiabaticindex"]
        if p["adiabatic"]:
            self.cs = torch.sqrt(g * (g - 1) * self.energy[:-1] / self.dens[:-1])
        done, n = 0.0, 0
        while done < 0.999999999 * DT:
            step = (DT - done) / self._limit(DT - done)
            done += step
            self._substep(step)
            n += 1
        return n

    def _substep(self, dt):
        p = self.p
        taper = 0.0 if self.t == 0 else 1.0  # the planet's mass grows within the first 1e-7 orbits
        mark = self._orbit()[1] if p["corotating"] else None
        sx, sy = self._pull(0.0, 0.0, 0.0)
        x0, y0 = self.pl[:2]
        d0, m = math.hypot(x0, y0), self.m * taper
        eps = p["thicknesssmoothing"] * p["aspectratio"] * d0
        pot = -m / torch.sqrt((self.x - x0) ** 2 + (self.y - y0) ** 2 + eps * eps) + m / d0 ** 3 * (self.x * x0 + self.y * y0)
        pot += -1 / self.rm + sx * self.x + sy * self.y
        if self.feels:
            gx, gy = self._pull(x0, y0, eps)
            self.pl[2] += dt * (gx - sx)
            self.pl[3] += dt * (gy - sy)
        self._advance_planet(dt)
        if mark is not None:
            c = self._orbit()[1]
            om = math.asin((mark[0] * c[1] - c[0] * mark[1]) / (math.hypot(*c) * math.hypot(*mark))) / dt
            self.vtheta[:-1] -= (om - self.om) * self.rm
            self.om = om
        c, s = math.cos(self.om * dt), math.sin(self.om * dt)
        x, y, vx, vy = self.pl
        self.pl = [x * c + y * s, -x * s + y * c, vx * c + vy * s, -vx * s + vy * c]
        self._boundary()
        self._source(dt, pot)
        self._boundary()
        if p["adiabatic"]:
            self._heat(dt)
        self._transport(dt)
        self._boundary()
        if p["adiabatic"]:
            self.temperature[:-1] = (p["adiabaticindex"] - 1) * self.energy[:-1] / self.dens[:-1]
        else:
            self.temperature[:-1] = self.pressure / self.dens[:-1]
        self.t += dt

    def _boundary(self):
        """The non-reflecting rings, with what the scheme's own threads past the ring's end write into rings 2 and nrad."""
        if not self.p["non_reflecting"]:
            return
        nr, ns, g = self.nr, self.ns, self.p["adiabaticindex"]
        D, E, V = self.dens, self.energy, self.vrad
        self.cs = cs = torch.sqrt(g * (g - 1) * E[:-1] / D[:-1])
        mean = cs.mean(1)

        def shift(k, ring):
            w = (float(self.r[k, 0]) ** -1.5 - 1) / (0.5 * float(mean[ring] + mean[ring - 1])) * float(self.rm[ring, 0] - self.rm[ring - 1, 0])
            return int(w / 2 / math.pi * ns + 0.5)

        first, last = shift(1, 1), shift(nr - 2, nr - 1)
        for F in (D, E):
            F[0] = torch.roll(F[1], first)
            F[nr - 1] = torch.roll(F[nr - 2], last)
        s1, s2 = float(self.smed[1, 0]), float(self.smed[nr - 2, 0])
        over = (1 << (ns - 1).bit_length()) - ns
        V[1] = 2 * (-cs[1] * (D[1] - s1) / s1) - V[2]
        V[nr - 1] = 2 * (cs[nr - 1] * (D[nr - 2] - s2) / s2) - V[nr - 2]
        if over:
            V[2, :over] = 2 * (-cs[2, :over] * (D[2, :over] - s1) / s1) - V[3, :over]
            V[nr, :over] = -V[nr - 1, :over]  # the sound speed past the last ring is zero
        for F, med in ((D, self.smed), (E, self.emed)):
            F[0] += med[0] - F[0].mean()
            F[nr - 1] += med[nr - 1] - F[nr - 1].mean()

    def _stress(self, vr, vt):
        """Divergence and stresses tau_rr, tau_phiphi at the centres, tau_rphi at the corners (zero on ring 0)."""
        d, nu = self.dens[:-1], self.nu
        up = (torch.roll(vt, -1, 1) - vt) / self.dphi / self.rm
        drr = (vr[1:] - vr[:-1]) / (self.rs - self.ri)
        dpp = up + 0.5 * (vr[1:] + vr[:-1]) / self.rm
        div = (vr[1:] * self.rs - vr[:-1] * self.ri) / (self.rs - self.ri) / self.rm + up
        w = vt / self.rm
        drp = 0.5 * (self.ri[1:] * (w[1:] - w[:-1]) / self.drm + (vr[1:-1] - torch.roll(vr[1:-1], 1, 1)) / self.dphi / self.ri[1:])
        ds = d[1:] + d[:-1]
        trp = torch.zeros_like(d)
        trp[1:] = 0.5 * (ds + torch.roll(ds, 1, 1)) * nu[1:] * drp
        return div, 2 * d * nu * (drr - div / 3), 2 * d * nu * (dpp - div / 3), trp

    def _source(self, dt, pot):
        p, d, vt = self.p, self.dens[:-1], self.vtheta[:-1]
        pr = (p["adiabaticindex"] - 1) * self.energy[:-1] if p["adiabatic"] else d * self.cs * self.cs
        self.pressure = pr
        self.nu = self._nu(self.cs)
        vr = torch.zeros_like(self.vrad)
        four = vt + torch.roll(vt, -1, 1)
        av = (four[1:] + four[:-1]) / 4 + self.om * self.ri[1:]
        sr, st = d[1:] + d[:-1], d + torch.roll(d, 1, 1)
        vr[1:-1] = self.vrad[1:-1] + dt * (-(pr[1:] - pr[:-1]) * 2 / sr / self.drm - (pot[1:] - pot[:-1]) / self.drm + av * av / self.ri[1:])
        vt = vt - dt * ((pr - torch.roll(pr, 1, 1)) * 2 / st + pot - torch.roll(pot, 1, 1)) / self.dx
        if p["self_gravity"]:
            ar, at = self._gravity(d)
            vr[1:-1] += dt * ((self.ri[1:] - self.rm[:-1]) * ar[1:] + (self.rm[1:] - self.ri[1:]) * ar[:-1]) / self.drm
            prev = torch.cat([torch.zeros(1, dtype=at.dtype, device=self.dev), at.reshape(-1)[:-1]]).view_as(at)  # flat: sector 0 takes the ring before
            vt += 0.5 * dt * (at + prev)
        _, trr, tpp, trp = self._stress(vr, vt)
        mid = slice(1, -1)
        vt[mid] += dt / self.rm[mid] * ((self.rs[mid] * trp[2:] - self.ri[mid] * trp[mid]) / (self.rs - self.ri)[mid] +
                                        (tpp - torch.roll(tpp, 1, 1))[mid] / self.dphi + 0.5 * (trp[mid] + trp[2:])) / (0.5 * st[mid])
        vr[1:-1] += dt / self.ri[1:] * ((self.rm[1:] * trr[1:] - self.rm[:-1] * trr[:-1]) / self.drm + (torch.roll(trp, -1, 1) - trp)[1:] / self.dphi -
                                        0.5 * (tpp[1:] + tpp[:-1])) / (0.5 * sr)
        edge = self.vkep2 - (self.rm * self.cs.mean(1, keepdim=True) if p["self_gravity"] else 0)
        for k in (0, -1):
            vt[k] = torch.sqrt(edge[k]) - self.rm[k] * self.om
        # artificial viscosity
        dr, dt_ = vr[1:] - vr[:-1], torch.roll(vt, -1, 1) - vt
        c2 = 1.41 * 1.41
        qr, qt = torch.where(dr < 0, c2 * d * dr * dr, 0.0), torch.where(dt_ < 0, c2 * d * dt_ * dt_, 0.0)
        self.vrad = torch.zeros_like(vr)
        self.vrad[1:-1] = vr[1:-1] - dt * 2 / sr * (qr[1:] - qr[:-1]) / self.drm
        self.vtheta = torch.nn.functional.pad(vt - dt * 2 / st * (qt - torch.roll(qt, 1, 1)) / self.dx, (0, 0, 0, 1))
        if p["adiabatic"]:
            self.eint = self.energy[:-1] - dt * qr * dr / (self.rs - self.ri) - dt * qt * dt_ / self.dx

    def _heat(self, dt):
        p, d, g = self.p, self.dens[:-1], self.p["adiabaticindex"]
        self.nu = nu = self._nu(self.cs)
        div, trr, tpp, trp = self._stress(self.vrad, self.vtheta[:-1])
        q = 0.5 / nu / d * (trr ** 2 + trp ** 2 + tpp ** 2) + 2 / 9 * nu * d * div * div
        lr = torch.log(self.rm[:3, 0])
        q[0] = q[1] * torch.exp(torch.log(q[1] / q[2]) * (lr[0] - lr[1]) / (lr[1] - lr[2]))
        if not p["cooling"]:
            new = (dt * q + self.eint) / (1 + (g - 1) * dt * div)
        else:
            tc = self.tcool
            new = (self.emed * dt * d / self.smed + tc * self.eint + dt * tc * (q - self.qmed * d / self.smed)) / (dt + tc + (g - 1) * dt * tc * div)
        self.energy[:-1] = new

    def _transport(self, dt):
        """Van Leer's scheme on momenta, energy and density: radially, then in azimuth about the ring's mean, shifted by whole sectors."""
        p, d, vr, vt, rm = self.p, self.dens[:-1], self.vrad, self.vtheta[:-1], self.rm
        qs = [d * vr[1:], d * vr[:-1], d * (torch.roll(vt, -1, 1) + rm * self.om) * rm, d * (vt + rm * self.om) * rm]
        qs += ([self.energy[:-1]] if p["adiabatic"] else []) + [d]
        zero = torch.zeros((1, self.ns), dtype=d.dtype, device=self.dev)
        v = vr[1:-1]  # the inner interfaces

        def limited(a, b):
            return torch.where(a * b > 0, a * b / torch.where(a * b > 0, a + b, 1.0), 0.0)

        def star_r(q):
            s = (q[1:] - q[:-1]) / self.drm
            dq = torch.cat([zero, 2 * limited(s[1:], s[:-1]), zero])
            rext = torch.cat([rm, torch.zeros_like(rm[:1])])
            up = q[:-1] + (self.drm - v * dt) * 0.5 * dq[:-1]
            dn = q[1:] - (rext[2:] - rm[1:] + v * dt) * 0.5 * dq[1:]
            return torch.where(v > 0, up, dn)

        flux = dt * self.dphi * self.ri[1:] * star_r(d) * v
        for k, q in enumerate(qs):
            f = torch.cat([zero, star_r(q / (d + 1e-20)) * flux, zero])
            qs[k] = q + (f[:-1] - f[1:]) / self.surf
        mean = vt.mean(1, keepdim=True)
        n = mean / rm * dt * self.ns / 2 / math.pi
        whole = torch.floor(n + 0.5)
        qs = self._sweep(qs, vt - mean, dt, limited)
        qs = self._sweep(qs, ((n - whole) * rm / dt * self.dphi).expand_as(vt), dt, limited)
        at = (torch.arange(self.ns, device=self.dev)[None] - whole.long()) % self.ns
        qs = [torch.gather(q, 1, at) for q in qs]
        d = qs[-1]
        self.dens = torch.nn.functional.pad(d, (0, 0, 0, 1))
        if p["adiabatic"]:
            self.energy = torch.nn.functional.pad(qs[4], (0, 0, 0, 1))
        self.vrad[0] = 0
        self.vrad[1:-1] = (qs[0][:-1] + qs[1][1:]) / (d[1:] + d[:-1] + 1e-20)
        self.vtheta[:-1] = (torch.roll(qs[2], 1, 1) + qs[3]) / (d + torch.roll(d, 1, 1) + 1e-15) / rm - rm * self.om

    def _sweep(self, qs, v, dt, limited):
        ksi = v * dt

        def star(q):
            s = torch.roll(q, -1, 1) - q
            dq = limited(s, torch.roll(s, 1, 1)) / self.dx
            return torch.where(ksi > 0, torch.roll(q, 1, 1) + (self.dx - ksi) * torch.roll(dq, 1, 1), q - (self.dx + ksi) * dq)

        d = qs[-1]
        flux = (self.rs - self.ri) * ksi * star(d)
        out = []
        for q in qs:
            f = star(q / (d + 1e-20)) * flux
            out.append(q + (f - torch.roll(f, -1, 1)) / self.surf)
        return out

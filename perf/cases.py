"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case goes through the public Python entry points (fsibe_2d_gb300.Run and Ensemble).  A
case is a dict of plain values; its "kind" says which calls it stands for:

  coupled    the time loop of the coupled solver: mask, fluid step, forces, beam, advance, from the
             captured step graph, with the per-step rows and the final fields read back at the end
  single     the same loop driven step by step by a host program that reads each step's scalars
  driver     the reference driver's own routine calls, one after another, every step
  obstacle   the fluid past a prescribed rigid obstacle (the mask uploaded by the caller)
  gradient   the adjoint: the gradient of the mean drag past a rigid obstacle
  ensemble   many runs of uneven sizes advanced together
  transform  the packed 2-D transforms on host arrays, forward and back

The FP32-compensated form's fields are single precision, so a program that runs it keeps them
in single precision, and so do these cases; the FP64 form's are returned as they are.
"""
import math

import numpy as np
import torch

import fsibe_2d_gb300 as F

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one step at a time on the smoke test's grid, its scalars read after
        # each, as a host program that steers the run does; bound by latency and launches
        dict(name="single_64_fp64", kind="single", nx=64, ny=64, ns=16, precision="fp64", Re=100.0, EI=0.1, mu=1.0,
             dt=2e-4, steps=4),
        # the plain FP64 run of the reference: 256^2, ns = 64
        dict(name="coupled_256_fp64", kind="coupled", nx=256, ny=256, ns=64, precision="fp64", Re=100.0, EI=0.1, mu=1.0,
             dt=2e-4, steps=100),
        # the headline workload, FP32-compensated, and the FP64 form on the same problem
        dict(name="coupled_1024_fp32", kind="coupled", nx=1024, ny=1024, ns=256, precision="fp32", Re=500.0, EI=0.1,
             mu=1.0, dt=5e-5, steps=100),
        dict(name="coupled_1024_fp64", kind="coupled", nx=1024, ny=1024, ns=256, precision="fp64", Re=500.0, EI=0.1,
             mu=1.0, dt=5e-5, steps=20),
        # the large single run: fields beyond L2, the longest beam
        dict(name="coupled_4096_fp32", kind="coupled", nx=4096, ny=4096, ns=1024, precision="fp32", Re=2000.0, EI=0.05,
             mu=2.0, dt=1e-5, steps=60, xl=8.0, eps=1e-4, band=32),
        # a channel: walls, leading-edge cylinder and a non-square grid, an odd number of beam nodes
        dict(name="channel_512x256_fp64", kind="coupled", nx=512, ny=256, ns=101, precision="fp64", Re=200.0, EI=0.2,
             mu=1.0, dt=1e-4, steps=40, walls=0.2, cylinder=0.06),
        # a heaving leading edge with the vorticity sponge and every per-step record kept
        dict(name="heaving_512_fp32", kind="coupled", nx=512, ny=512, ns=127, precision="fp32", Re=300.0, EI=0.1, mu=2.0,
             dt=1e-4, steps=100, motion=305, sponge=3, records=True),
        # the reference driver's call sequence (time_step.f90), routine by routine
        dict(name="driver_512_fp32", kind="driver", nx=512, ny=512, ns=128, precision="fp32", Re=200.0, EI=0.1, mu=1.0,
             dt=1e-4, steps=20),
        # flow past a rigid obstacle without a flexible beam
        dict(name="obstacle_2048_fp32", kind="obstacle", nx=2048, ny=2048, ns=65, precision="fp32", Re=500.0, dt=2.5e-5,
             steps=100, angle=10.0),
        # the adjoint configuration's grid: forward and reverse steps with binomial checkpointing
        dict(name="gradient_512_fp64", kind="gradient", nx=512, ny=512, ns=128, precision="fp64", Re=200.0, dt=1e-4,
             steps=40, snapshots=8, angle=10.0),
        # the batched configuration: 48 x 256^2, 12 x 512^2 and 4 x 1024^2
        dict(name="ensemble_64_fp32", kind="ensemble", n256=48, n512=12, n1024=4, precision="fp32", dt=5e-5, steps=40),
        # the transforms called on host arrays (coftxy / cofitxy)
        dict(name="transform_512x1024_fp64", kind="transform", nx=1024, ny=512, precision="fp64"),
    ]


def draw(rng):
    kind = rng.choice(["coupled", "coupled", "coupled", "single", "driver", "obstacle", "gradient", "ensemble", "transform"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "ensemble":
        return dict(kind=kind, n256=rng.randint(4, 40), n512=rng.randint(1, 10), n1024=rng.randint(0, 3), precision="fp32",
                    dt=5e-5, steps=rng.randint(5, 30))
    top = {"coupled": 12, "single": 9, "driver": 11, "obstacle": 11, "gradient": 9, "transform": 11}[kind]
    lx = rng.randint(6, top)
    if prec == "fp64":
        lx = min(lx, 11)
    nx = 1 << lx
    ny = nx >> rng.choice([0, 0, 1])
    if kind == "transform":
        return dict(kind=kind, nx=nx, ny=ny, precision=prec)
    if kind == "gradient":
        prec = "fp64"
    c = dict(kind=kind, nx=nx, ny=ny, ns=rng.randint(max(9, nx // 8), max(17, nx // 4)), precision=prec,
             Re=round(rng.uniform(100.0, 1000.0), 3), dt=min(2e-4, 0.0128 * 4.0 / nx))
    # as many steps as some 5 to 50 ms hold (about 0.2 ms and 0.1 or 1 ns a cell each)
    ms = math.exp(rng.uniform(math.log(5.0), math.log(50.0)))
    per = 0.2 + nx * ny * (1e-6 if prec == "fp64" else 1e-7)
    c["steps"] = max(3, min(200, int(ms / per)))
    if kind in ("obstacle", "gradient"):
        c["angle"] = round(rng.uniform(5.0, 20.0), 3)
        if kind == "gradient":
            c["steps"] = max(6, c["steps"] // 5)
            c["snapshots"] = rng.randint(2, 12)
        return c
    c["EI"] = round(10.0 ** rng.uniform(-1.5, 0.0), 5)
    c["mu"] = round(rng.uniform(0.5, 5.0), 4)
    if kind == "single":
        c["steps"] = rng.randint(2, 12)
    elif kind == "coupled" and nx >= 128:
        option = rng.choice(["plain", "plain", "heaving", "walls", "sponge"])
        if option == "heaving":
            c["motion"] = rng.choice([2, 205, 305])
        elif option == "walls" and ny == nx:
            c["walls"] = 0.3
        elif option == "sponge":
            c["sponge"] = rng.choice([1, 2, 3])
        if rng.random() < 0.3:
            c["records"] = True
    return c


# ---- inputs ---------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _vorticity(nx, ny, gen, band=8, sigma=1e-3):
    """Seeded N(0, sigma) noise, low-passed to |k| <= band: the start field of the benchmark runs."""
    w = torch.randn((ny, nx), generator=gen, device=DEVICE, dtype=torch.float64) * sigma
    k = torch.fft.rfft2(w)
    kx = torch.arange(nx // 2 + 1, device=DEVICE, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, 1.0 / ny, device=DEVICE, dtype=torch.float64)
    k[(kx[None, :] ** 2 + ky[:, None] ** 2) > band * band] = 0.0
    return torch.fft.irfft2(k, s=(ny, nx)).cpu().numpy()


def _box(case):
    xl = case.get("xl", 4.0)
    return xl, xl * case["ny"] / case["nx"]


def _obstacle(case):
    """chi / eps of an inclined elliptic plate with a smooth edge two cells wide."""
    nx, ny = case["nx"], case["ny"]
    xl, yl = _box(case)
    x = (np.arange(nx) * (xl / nx) - (0.25 * xl + 0.5))[None, :]
    y = (np.arange(ny) * (yl / ny) - 0.5 * yl)[:, None]
    a = math.radians(case["angle"])
    p, q = x * math.cos(a) + y * math.sin(a), -x * math.sin(a) + y * math.cos(a)
    b = max(0.05, 2.0 * xl / nx)
    d = (np.sqrt((p / 0.5) ** 2 + (q / b) ** 2) - 1.0) * b
    return 0.5 * (1.0 - np.tanh(d / (2.0 * xl / nx))) / case.get("eps", 1e-3)


def _params(case, **more):
    xl, yl = _box(case)
    kw = dict(nx=case["nx"], ny=case["ny"], ns=case.get("ns", 64), xl=xl, yl=yl, x0=0.25 * xl, y0=0.5 * yl,
              Re=case.get("Re", 100.0), eps=case.get("eps", 1e-3), dt=case.get("dt", 1e-4),
              EI=case.get("EI", 0.1), mu=case.get("mu", 1.0),
              precision=F.FSIBE_FP64 if case["precision"] == "fp64" else F.FSIBE_FP32C)
    if case.get("motion"):
        kw["iMotion"] = case["motion"]
    if case.get("walls"):
        kw.update(iWalls=1, h_channel=case["walls"])
    if case.get("cylinder"):
        kw.update(iCylinder=1, R_cylinder=case["cylinder"])
    if case.get("sponge"):
        kw.update(iSponge=case["sponge"], SpongeSize=0.1 * yl, eps_sponge=1e-2)
    kw.update(more)
    return F.make_params(**kw)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "ensemble":
        rng = np.random.default_rng(seed)
        ps = []
        for n in (256, 512, 1024):
            for _ in range(case["n%d" % n]):
                ps.append(F.make_params(nx=n, ny=n, ns=n // 4, precision=F.FSIBE_FP32C, dt=case["dt"],
                                        Re=float(rng.uniform(100, 1000)), EI=float(10 ** rng.uniform(-2, 0)),
                                        mu=float(rng.uniform(0.5, 5))))
        ens = F.Ensemble(ps)
        for r, p in zip(ens.runs, ps):
            r.init_fields(_vorticity(p.nx, p.ny, gen))
        return dict(case=case, ens=ens)
    if kind == "transform":
        f = torch.randn((case["ny"], case["nx"]), generator=gen, device=DEVICE, dtype=torch.float64).cpu().numpy()
        return dict(case=case, run=F.Run(_params(case)), field=f)
    w = _vorticity(case["nx"], case["ny"], gen, band=case.get("band", 8), sigma=1e-2 if kind == "gradient" else 1e-3)
    if kind in ("obstacle", "gradient"):
        # a beam that does not move (its nodes give the drag's window), the mask from the caller
        r = F.Run(_params(case, iFLUSI=0, iMotion=0, angle_beam=case["angle"], cfl=10.0,
                          iSaveBeam=0 if kind == "gradient" else 3))
        m = _obstacle(case)
        zero = np.zeros_like(m)
        r.init_fields(w)
        r.set_mask(m, zero, zero)
        if kind == "obstacle":
            r.use_graph(True)
        return dict(case=case, run=r, vort=w)
    r = F.Run(_params(case))
    if kind != "driver":
        r.use_graph(True)
    r.init_fields(w)
    return dict(case=case, run=r, started=False)


# ---- one pass -------------------------------------------------------------------------------

def _kept(case, a):
    """What a program keeps of a result: single precision for the FP32-compensated form."""
    return a.astype(np.float32) if case["precision"] == "fp32" else a


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        ens = state["ens"]
        ens.step(case["steps"])
        out = {"rows": _kept(case, np.array([list(r.scalars().beam_data) for r in ens.runs])),
               "beams": _kept(case, np.concatenate([r.beam()[0].reshape(-1) for r in ens.runs]))}
        for n in (256, 512, 1024):
            w = [_kept(case, r.vort()) for r in ens.runs if r.nx == n]
            if w:
                out["vort%d" % n] = np.stack(w)
        return out
    r = state["run"]
    if kind == "transform":
        fk = r.coftxy(state["field"])
        return {"packed": _kept(case, fk), "back": _kept(case, r.cofitxy(fk))}
    if kind == "gradient":
        J, gv, gm, gnu, _ = r.drag_gradient(state["vort"], case["steps"], case["steps"] // 2 + 1,
                                            snapshots=case["snapshots"])
        return {"J": J, "g_vort": gv, "g_mask": gm, "g_nu": gnu}
    if kind == "obstacle":
        r.time_step(case["steps"])
        return {"vort": _kept(case, r.vort()), "u": _kept(case, r.u()), "press": _kept(case, r.press())}
    if kind == "single":
        rows = []
        for _ in range(case["steps"]):
            r.step()
            rows.append(list(r.scalars().beam_data))
        rows = np.array(rows)
    elif kind == "driver":
        t = r.scalars().time
        rows = []
        for _ in range(case["steps"]):
            if state["started"]:
                r.create_mask(t)
                r.EvolveFluidAB2()
            else:
                r.create_mask(t)
                r.EvolveFluidExplicit()
                state["started"] = True
            r.GetForces(t)
            r.SolidSolverWrapper(t)
            r.advance()
            s = r.scalars()
            t = s.time
            rows.append(list(s.beam_data))
        rows = np.array(rows)
    elif case.get("records"):
        rows = r.run_records(case["steps"])
    else:
        rows = r.time_step(case["steps"])
    return {"rows": _kept(case, rows), "beam": _kept(case, r.beam()[0]), "vort": _kept(case, r.vort())}


# ---- what a pass cannot do without ----------------------------------------------------------

def _step_work(nx, ny, fp32, coupled):
    """One time step: the state (the vorticity, its AB2 history, the velocity, the mean vorticity and
    the mask with its velocity) read once and written once; twelve real 2-D transforms and some
    eighty operations a cell."""
    cells = nx * ny
    fields = (6 if fp32 else 5) * 2 + (6 if coupled else 3)
    return fields * cells * (4 if fp32 else 8), cells * (12 * 2.5 * math.log2(cells) + 80.0)


def work(case):
    kind = case["kind"]
    fp32 = case["precision"] == "fp32"
    size = 4 if fp32 else 8
    if kind == "ensemble":
        b = f = 0.0
        for n in (256, 512, 1024):
            sb, sf = _step_work(n, n, True, True)
            b += case["n%d" % n] * (case["steps"] * sb + 4 * n * n)
            f += case["n%d" % n] * case["steps"] * sf
        return {"bytes": b, "flops": f}
    nx, ny = case["nx"], case["ny"]
    cells = nx * ny
    if kind == "transform":
        return {"bytes": 4.0 * 8 * cells, "flops": 2 * 2.5 * cells * math.log2(cells)}
    sb, sf = _step_work(nx, ny, fp32, kind not in ("obstacle", "gradient"))
    n = case["steps"]
    if kind == "gradient":
        # a forward step and a reverse step of about twice its work each
        return {"bytes": 3.0 * n * sb + 4 * 8 * cells, "flops": 3.0 * n * sf}
    return {"bytes": float(n * sb + size * cells * (4 if kind == "obstacle" else 1)), "flops": float(n * sf)}


# ---- the same in 64 bits, by torch alone ----------------------------------------------------

class _Fluid:
    """The fluid step on a fixed mask at rest: spectra of rfft2 / (nx ny) with the Nyquist modes removed."""

    def __init__(self, case, mask, nu):
        self.nx, self.ny = case["nx"], case["ny"]
        xl, yl = _box(case)
        self.dx, self.dy = xl / self.nx, yl / self.ny
        self.dt = min(case["dt"], 0.9 * case.get("eps", 1e-3))
        kx = torch.arange(self.nx // 2 + 1, device=DEVICE, dtype=torch.float64)[None, :]
        ky = torch.fft.fftfreq(self.ny, 1.0 / self.ny, device=DEVICE, dtype=torch.float64)[:, None]
        self.keep = ((kx < self.nx // 2) & (ky.abs() < self.ny // 2)).to(torch.float64)
        self.ikx, self.iky = 1j * kx * (2 * math.pi / xl), 1j * ky * (2 * math.pi / yl)
        k2 = (kx * 2 * math.pi / xl) ** 2 + (ky * 2 * math.pi / yl) ** 2
        self.k2 = k2
        self.inv_k2 = torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
        kxt, kyt = 2.0 / 3.0 * (self.nx // 2 - 1), 2.0 / 3.0 * (self.ny // 2 - 1)
        self.dealias = ((kx * kx / (kxt * kxt) + ky * ky / (kyt * kyt)) < 1.0).to(torch.float64) * self.keep
        self.mask = mask
        self.E = torch.exp(-nu * self.dt * k2)

    def fwd(self, f):
        return torch.fft.rfft2(f) * (self.keep / (self.nx * self.ny))

    def inv(self, s):
        return torch.fft.irfft2(s * (self.nx * self.ny), s=(self.ny, self.nx))

    def velocity(self, w):
        psi = w * self.inv_k2
        return self.inv(self.iky * psi) + 1.0, -self.inv(self.ikx * psi)

    def step(self, w, hist, u, v):
        n = self.fwd(-u * self.inv(self.ikx * w) - v * self.inv(self.iky * w))
        n = n - self.ikx * self.fwd(self.mask * v) + self.iky * self.fwd(self.mask * u)
        new = w + self.dt * n if hist is None else w + 1.5 * self.dt * n - 0.5 * self.dt * hist
        w = new * self.E * self.dealias
        u, v = self.velocity(w)
        return w, n * self.E, u, v

    def pressure(self, w, u, v):
        om = self.inv(w)
        q = self.ikx * self.fwd(self.mask * u - om * v) + self.iky * self.fwd(self.mask * v + om * u)
        return self.inv(q * self.inv_k2) - 0.5 * (u * u + v * v)


def _window(case):
    """The cells of the drag's sum, from the straight beam's nodes (1.5 half thicknesses around them)."""
    xl, yl = _box(case)
    dx, dy = xl / case["nx"], yl / case["ny"]
    a, tb = math.radians(case["angle"]), 2.0 * dx
    xs, ys = (0.25 * xl, 0.25 * xl + math.cos(a)), (0.5 * yl, 0.5 * yl + math.sin(a))
    x0, x1 = int((min(xs) - 1.5 * tb) / dx), int((max(xs) + 1.5 * tb) / dx)
    y0, y1 = int((min(ys) - 1.5 * tb) / dy), int((max(ys) + 1.5 * tb) / dy)
    return max(x0, 0), min(x1, case["nx"] - 1), max(y0, 0), min(y1, case["ny"] - 1)


def _packed(f):
    """coftxy's packed layout of the normalised transform, Nyquist modes removed."""
    ny, nx = f.shape
    h = nx // 2
    ft = np.fft.fft(np.fft.rfft(f, axis=1)[:, :h], axis=0) / (nx * ny)
    out = np.zeros((ny, nx))
    out[0, 0::2], out[0, 1::2] = ft[0].real, ft[0].imag
    j = np.arange(1, ny // 2)
    p, m = ft[j], ft[ny - j]
    out[2 * j, 0::2], out[2 * j + 1, 0::2] = 0.5 * (p.real + m.real), 0.5 * (p.imag - m.imag)
    out[2 * j, 1::2], out[2 * j + 1, 1::2] = 0.5 * (p.imag + m.imag), 0.5 * (m.real - p.real)
    return out


def exact(case, seed):
    """The fluid alone and the transforms; the coupled runs have no short restatement."""
    kind = case["kind"]
    if kind not in ("obstacle", "gradient", "transform"):
        return None
    gen = _generator(seed)
    if kind == "transform":
        f = torch.randn((case["ny"], case["nx"]), generator=gen, device=DEVICE, dtype=torch.float64).cpu().numpy()
        ft = np.fft.rfft2(f)
        ft[:, -1] = 0.0
        ft[case["ny"] // 2] = 0.0
        return {"packed": _packed(f), "back": np.fft.irfft2(ft, s=f.shape)}
    w0 = torch.from_numpy(_vorticity(case["nx"], case["ny"], gen, band=case.get("band", 8),
                                     sigma=1e-2 if kind == "gradient" else 1e-3)).to(DEVICE)
    m = torch.from_numpy(_obstacle(case)).to(DEVICE)
    if kind == "obstacle":
        fl = _Fluid(case, m, 1.0 / case["Re"])
        w, hist = fl.fwd(w0), None
        u, v = fl.velocity(w)
        for _ in range(case["steps"]):
            w, hist, u, v = fl.step(w, hist, u, v)
        return {"vort": fl.inv(w).cpu().numpy(), "u": torch.stack([u, v]).cpu().numpy(),
                "press": fl.pressure(w, u, v).cpu().numpy()}
    w0.requires_grad_(True)
    m.requires_grad_(True)
    nu = torch.tensor(1.0 / case["Re"], device=DEVICE, dtype=torch.float64, requires_grad=True)
    fl = _Fluid(case, m, nu)
    x0, x1, y0, y1 = _window(case)
    w, hist = fl.fwd(w0), None
    u, v = fl.velocity(w)
    J, first = 0.0, case["steps"] // 2 + 1
    for k in range(1, case["steps"] + 1):
        w, hist, u, v = fl.step(w, hist, u, v)
        if k >= first:
            J = J + (m * u)[y0:y1 + 1, x0:x1 + 1].sum() * (fl.dx * fl.dy)
    J = J / (case["steps"] - first + 1)
    J.backward()
    return {"J": float(J.detach()), "g_vort": w0.grad.cpu().numpy(), "g_mask": m.grad.cpu().numpy(),
            "g_nu": float(nu.grad)}

"""What the framework is timed on: the work its users have it do, through its public entry points.

A case is one pass of a user's program on a solver, an ensemble, a server or a generic-shape
grid that the program keeps: some RK3 steps (or one transform), then the result it reads.
Sizes are the repository's own: the grids of its tests (8 .. 128, with the 3 * 2^k ones), the
published benchmark grids (64, 128, 256), the bench grid (512), the ensemble's and the serving
stream's mixes, and boxes off the benchmark domain.  Everything starts from the Taylor-Green
field plus the framework's seeded perturbation, at Reynolds numbers of the serving stream.

A solve ends with the whole physical velocity in pinned host memory, as a program writes its
snapshots; the FP32 precision form's snapshots are kept in float32, the precision it
computes in.  The spectral divergence column of the diagnostics is left out: it is zero but
for round-off.
"""
import ctypes
import math

import numpy as np
import torch

from spectral_solver_b200 import Batch, Fft3D, Server, Solver, load

TWO_PI = 2.0 * math.pi
AMP = 0.05  # rms of the seeded perturbation: a visibly disturbed Taylor-Green vortex
CFL = 0.3
ROW = ("kinetic_energy", "dissipation", "enstrophy", "max_velocity")


# ---------------------------------------------------------------------------------------
# The cases
def listed():
    return [
        # the smallest call: one forward transform of a device field, on the caller's buffers
        dict(name="forward48", kind="forward", n=48),
        # the published FP64 benchmark's loop on its 64^3 grid: vmax, the CFL step, the step,
        # from the host at every step, and a diagnostics row at the end
        dict(name="loop64_fp64", kind="solve", n=64, fp32=False, stepping="loop", steps=40, re=1600.0),
        # a small grid that is not a power of two, integrating-factor viscosity, precision form
        dict(name="if48_fp32", kind="solve", n=48, fp32=True, stepping="fixed", steps=100, re=800.0, visc_if=True),
        # the CFL step taken on the device, FP64, a 3 * 2^k grid
        dict(name="cfl96_fp64", kind="solve", n=96, fp32=False, stepping="cfl", steps=40, re=1600.0),
        # the rotational form, which some users prefer for its robustness
        dict(name="rot128_fp64", kind="solve", n=128, fp32=False, stepping="fixed", steps=30, re=1600.0,
             rotational=True),
        # production runs of the middle grid: FP64 at a fixed step, FP32 at the CFL step
        dict(name="step256_fp64", kind="solve", n=256, fp32=False, stepping="fixed", steps=40, re=1600.0),
        dict(name="cfl256_fp32", kind="solve", n=256, fp32=True, stepping="cfl", steps=60, re=1600.0),
        # the headline workload in both forms: 512^3 at a fixed step
        dict(name="step512_fp32", kind="solve", n=512, fp32=True, stepping="fixed", steps=16, re=1600.0),
        dict(name="step512_fp64", kind="solve", n=512, fp32=False, stepping="fixed", steps=10, re=1600.0),
        # a parameter study: uneven solves stepped together, one graph launch per step
        dict(name="ensemble_fp32", kind="ensemble", fp32=True, steps=20,
             sizes="32 32 32 48 48 48 64 64 64 64 96 96 96 96 128 128 128 128"),
        # a short burst of the serving stream (its sizes and probabilities), to the last result
        dict(name="serve_fp32", kind="serve", fp32=True, sizes="64 128 64 64 256 64 128 64 128 64", t_end=0.3),
        # the reference's class on a domain off the benchmark's: an anisotropic box
        dict(name="box_96x80x60", kind="box", nx=96, ny=80, nz=60, lx=6.0, ly=5.0, lz=4.0, dealias=True, steps=6),
    ]


def draw(rng):
    kind = rng.choices(["forward", "solve", "ensemble", "serve", "box"], [1, 5, 1, 1, 2])[0]
    fp32 = rng.random() < 0.5
    if kind == "forward":
        return dict(kind=kind, n=rng.choice([8, 12, 16, 24, 32, 48, 64]))
    if kind == "solve":
        n = rng.choice([16, 24, 32, 48, 64, 96, 128, 256, 256, 512])
        most = {512: 16 if fp32 else 10, 256: 60 if fp32 else 40}.get(n, 100)
        form = rng.choices(["plain", "if", "rotational"], [4, 1, 1])[0]
        c = dict(kind=kind, n=n, fp32=fp32, stepping=rng.choice(["fixed", "cfl", "loop"]),
                 steps=rng.randint(most // 2, most), re=round(math.exp(rng.uniform(math.log(400), math.log(3200))), 1))
        if form == "if":
            c["visc_if"] = True
        if form == "rotational" and n < 512:
            c["rotational"] = True
        return c
    if kind == "ensemble":
        sizes = [rng.choice([16, 24, 32, 48, 64, 96, 128]) for _ in range(rng.randint(4, 24))]
        return dict(kind=kind, fp32=fp32, steps=rng.randint(8, 20), sizes=" ".join(map(str, sizes)))
    if kind == "serve":
        sizes = rng.choices([64, 128, 256], [6, 3, 1], k=rng.randint(3, 10))
        return dict(kind=kind, fp32=fp32, sizes=" ".join(map(str, sizes)), t_end=round(rng.uniform(0.1, 0.3), 3))
    pick = lambda: rng.choice([12, 17, 24, 30, 33, 45, 48, 64, 70, 72, 90, 96, 100])  # noqa: E731
    return dict(kind=kind, nx=pick(), ny=pick(), nz=pick(), lx=round(rng.uniform(1, 7), 3),
                ly=round(rng.uniform(1, 7), 3), lz=round(rng.uniform(1, 7), 3), dealias=rng.random() < 0.7,
                steps=rng.randint(2, 6))


# ---------------------------------------------------------------------------------------
# What a program has in hand, and one pass of it
class Snapshot:
    """The velocity of a solver, copied to pinned host memory at each call."""

    def __init__(self, n, fp32):
        self.buf = torch.empty(3, n, n, n, dtype=torch.float64, pin_memory=True)
        self.low = torch.empty(3, n, n, n, dtype=torch.float32).fill_(0.0) if fp32 else None
        self.ptrs = (ctypes.POINTER(ctypes.c_double) * 3)(
            *[ctypes.cast(self.buf[c].data_ptr(), ctypes.POINTER(ctypes.c_double)) for c in range(3)])

    def take(self, solver):
        rc = solver.lib.sns_dump_velocity(solver.h, self.ptrs)
        if rc:
            raise RuntimeError(solver.lib.sns_last_error(solver.h).decode())
        return self.buf if self.low is None else self.low.copy_(self.buf)


def kmax_of(n):
    return max(1, n // 8)


def dt_of(n):
    return 0.1 * TWO_PI / n


def prepare(case, seed):
    kind = case["kind"]
    if kind == "forward":
        n = case["n"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        phys = torch.randn(n, n, n, dtype=torch.float64, device="cuda", generator=gen)
        spec = torch.empty(n, n, n, dtype=torch.complex128, device="cuda")
        return dict(case=case, lib=load(), phys=phys, spec=spec)
    if kind == "solve":
        n = case["n"]
        s = Solver(n, case["re"], seed=seed, pert_amp=AMP, pert_kmax=kmax_of(n), precision=int(case["fp32"]),
                   viscous_mode=int(case.get("visc_if", False)))
        if case.get("rotational"):
            s.set_nonlinear_form(1)
        if case["stepping"] == "cfl":
            s.set_clock(0.0, cfl=CFL, dt_max=0.5)
        return dict(case=case, solver=s, snap=Snapshot(n, case["fp32"]))
    if kind == "ensemble":
        specs = [dict(sp, precision=int(case["fp32"]), dt=0.0, cfl=CFL, dt_max=0.5) for sp in members(case, seed)]
        b = Batch(specs)
        return dict(case=case, batch=b, solvers=[b.solver(i) for i in range(len(specs))],
                    snaps=[Snapshot(sp["n"], case["fp32"]) for sp in specs])
    if kind == "serve":
        return dict(case=case, server=Server(80_000_000_000, precision=int(case["fp32"])),
                    requests=[dict(sp, t_end=case["t_end"]) for sp in members(case, seed)])
    grid = Fft3D((case["nx"], case["ny"], case["nz"]), (case["lx"], case["ly"], case["lz"]))
    return dict(case=case, grid=grid, u=[c.cpu().numpy() for c in box_field(case, seed)])


def members(case, seed):
    """The solves of an ensemble or of a burst of requests: uneven N, Re and seed."""
    rng = np.random.default_rng(seed)
    return [dict(n=int(n), nu=1.0 / float(np.exp(rng.uniform(np.log(400.0), np.log(3200.0)))),
                 seed=int(rng.integers(1 << 40)), pert_amp=AMP, pert_kmax=kmax_of(int(n)))
            for n in case["sizes"].split()]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        rc = state["lib"].sns_forward_r2c_noalloc(case["n"], state["phys"].data_ptr(), state["spec"].data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(state["lib"].sns_last_error(None).decode())
        return state["spec"]
    if kind == "solve":
        s, steps = state["solver"], case["steps"]
        row = None
        if case["stepping"] == "fixed":
            s.step(dt_of(case["n"]), steps)
        elif case["stepping"] == "cfl":
            s.step_cfl(steps)
        else:
            dx = TWO_PI / case["n"]
            for _ in range(steps):
                s.step(min(0.5, CFL * dx / s.max_velocity()))
            d = s.diagnostics()
            row = [d[k] for k in ROW]
        out = dict(velocity=state["snap"].take(s))
        if row is not None:
            out["row"] = row
        return out
    if kind == "ensemble":
        state["batch"].step(case["steps"])
        return [snap.take(s) for snap, s in zip(state["snaps"], state["solvers"])]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(r["n"], r["nu"], r["t_end"], r["seed"], r["pert_amp"], r["pert_kmax"], CFL, 0.5)
               for r in state["requests"]]
        done = {}
        while len(done) < len(ids):
            for r in srv.step()[0]:
                done[r["id"]] = r
        return [dict(steps=done[i]["steps"], row=np.array([done[i]["final"][k] for k in ROW], dtype=np.float32))
                for i in ids]
    dt = 0.05 * min(case["lx"] / case["nx"], case["ly"] / case["ny"], case["lz"] / case["nz"])
    return state["grid"].step(state["u"], 1e-3, dt, case["steps"], dealias=case["dealias"])


# ---------------------------------------------------------------------------------------
# What a pass cannot do without: the state u read and written once per RK3 stage, g too after
# the first, and what is read at the end; the arithmetic of the 18 (9 without the phase-shift
# pair) real 3-D transforms of a stage.
def solve_work(n, fp32, steps, vmax_passes=0):
    w = 4 if fp32 else 8
    points = float(n) ** 3
    fft = 2.5 * points * math.log2(points)
    return (steps * points * w * 33.0,
            fft * (steps * 3 * 18 + vmax_passes * 3))


def work(case):
    kind = case["kind"]
    if kind == "forward":
        points = float(case["n"]) ** 3
        return dict(bytes=points * 24, flops=2.5 * points * math.log2(points))
    if kind == "solve":
        vm = case["steps"] if case["stepping"] != "fixed" else 0
        b, f = solve_work(case["n"], case["fp32"], case["steps"], vm)
        return dict(bytes=b + 24.0 * case["n"] ** 3, flops=f)
    if kind == "ensemble":
        parts = [solve_work(int(n), case["fp32"], case["steps"], case["steps"]) for n in case["sizes"].split()]
        out = sum(24.0 * int(n) ** 3 for n in case["sizes"].split())
        return dict(bytes=sum(p[0] for p in parts) + out, flops=sum(p[1] for p in parts))
    if kind == "serve":
        parts = []
        for n in map(int, case["sizes"].split()):
            steps = math.ceil(case["t_end"] / (CFL * TWO_PI / n))
            parts.append(solve_work(n, case["fp32"], steps, steps))
        return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))
    points = float(case["nx"] * case["ny"] * case["nz"])
    return dict(bytes=case["steps"] * points * 16 * 33 + 2 * 48 * points,
                flops=case["steps"] * 3 * (18 if case["dealias"] else 9) * 2.5 * points * math.log2(points))


# ---------------------------------------------------------------------------------------
# The same in 64 bits, from torch's FFTs alone
def splitmix64(x):
    with np.errstate(over="ignore"):
        z = x + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def perturbation(n, seed, amp, kmax):
    """Seeded solenoidal k^(-5/3) modes with 1 <= |m| <= kmax, as (iz, iy, ix) and values [3]."""
    r = np.arange(-kmax, kmax + 1)
    mz, my, mx = (a.reshape(-1) for a in np.meshgrid(r, r, np.arange(kmax + 1), indexing="ij"))
    k2 = mx * mx + my * my + mz * mz
    take = (k2 >= 1) & (k2 <= kmax * kmax) & ((mx > 0) | (my > 0) | ((my == 0) & (mz > 0)))
    mx, my, mz, k2 = mx[take], my[take], mz[take], k2[take].astype(np.float64)
    flat = (mx + n * ((my % n) + n * (mz % n))).astype(np.uint64)
    h = splitmix64(np.array([seed], dtype=np.uint64))
    v = []
    for c in range(3):
        bits = splitmix64(h ^ (np.uint64(3) * flat + np.uint64(c)))
        theta = (bits >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
        v.append(k2 ** (-5.0 / 6.0) * np.exp(1j * TWO_PI * theta))
    dot = (v[0] * mx + v[1] * my + v[2] * mz) / k2
    v = [v[0] - dot * mx, v[1] - dot * my, v[2] - dot * mz]
    total = sum(2.0 * np.abs(a) ** 2 for a in v).sum()
    v = [a * (amp / math.sqrt(total / float(n) ** 6)) for a in v]
    own = mx == 0  # the plane mx = 0 stores the mirror modes too
    at = [np.concatenate([a, (-a[own]) % n]) % n for a in (mz, my)] + [np.concatenate([mx, mx[own]])]
    return at, [np.concatenate([a, a[own].conj()]) for a in v]


class Exact:
    """The solve on the half spectrum [z][y][x <= n/2] in complex128."""

    def __init__(self, n, nu, seed, visc_if=False, rotational=False):
        self.n, self.nu, self.visc_if, self.rotational = n, nu, visc_if, rotational
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        i = torch.arange(n, dtype=torch.float64, device=dev)
        m = torch.where(i <= n // 2, i, i - n)
        mx, my, mz = i[: n // 2 + 1].view(1, 1, -1), m.view(1, -1, 1), m.view(-1, 1, 1)
        self.k = (mx, my, mz)
        self.k2 = mx * mx + my * my + mz * mz
        self.mask = 4.0 * self.k2 <= float(n * n)
        self.inv = torch.where(self.k2 > 0, 1.0 / self.k2.clamp(min=1.0), torch.zeros_like(self.k2)) * self.mask
        self.keep = (self.mask & (self.k2 > 0)).to(torch.float64)
        self.phase = torch.polar(torch.ones_like(self.k2), (mx + my + mz) * (math.pi / n))
        x = (i + 0.5) * TWO_PI / n
        X, Y, Z = x.view(1, 1, -1), x.view(1, -1, 1), x.view(-1, 1, 1)
        u = torch.fft.rfftn(torch.sin(X) * torch.cos(Y) * torch.cos(Z))
        v = torch.fft.rfftn(-torch.cos(X) * torch.sin(Y) * torch.cos(Z))
        self.u = [u, v, torch.zeros_like(u)]
        at, values = perturbation(n, seed, AMP, kmax_of(n))
        at = [torch.from_numpy(a.astype(np.int64)).to(dev) for a in at]
        for c in range(3):
            self.u[c][at[0], at[1], at[2]] += torch.from_numpy(values[c]).to(dev)
        self.project(self.u)
        self.g = [torch.zeros_like(u) for _ in range(3)]

    def project(self, f):
        dot = (f[0] * self.k[0] + f[1] * self.k[1] + f[2] * self.k[2]) * self.inv
        for c in range(3):
            f[c].sub_(dot * self.k[c]).mul_(self.keep)

    def real(self, f):
        return torch.fft.irfftn(f, s=(self.n,) * 3)

    def dealiased(self, a, b):
        a, b = torch.fft.rfftn(a), torch.fft.rfftn(b)
        return a.add_(b.mul_(self.phase.conj())).mul_(0.5).mul_(self.mask)

    def vorticity_hat(self):
        u, k = self.u, self.k
        return [1j * (k[(c + 1) % 3] * u[(c + 2) % 3] - k[(c + 2) % 3] * u[(c + 1) % 3]) for c in range(3)]

    def rhs(self):
        both = [[self.real(c) for c in self.u], [self.real(c * self.phase) for c in self.u]]
        if self.rotational:
            w = self.vorticity_hat()
            vort = [[self.real(c) for c in w], [self.real(c * self.phase) for c in w]]
            r = []
            for c in range(3):
                a, b = (c + 1) % 3, (c + 2) % 3
                p = [both[s][a] * vort[s][b] - both[s][b] * vort[s][a] for s in (0, 1)]
                r.append(self.dealiased(*p))
        else:
            r = [torch.zeros_like(self.u[0]) for _ in range(3)]
            for a in range(3):
                for b in range(a, 3):
                    p = self.dealiased(both[0][a] * both[0][b], both[1][a] * both[1][b]).mul_(-1j)
                    r[a].add_(p * self.k[b])
                    if a != b:
                        r[b].add_(p * self.k[a])
        if not self.visc_if:
            for c in range(3):
                r[c].sub_(self.u[c] * (self.nu * self.k2))
        self.project(r)
        return r

    def step(self, dt):
        for a, b, tau in ((0.0, dt / 3.0, dt / 3.0), (-5.0 / 9.0, 15.0 * dt / 16.0, 5.0 * dt / 12.0),
                          (-153.0 / 128.0, 8.0 * dt / 15.0, dt / 4.0)):
            r = self.rhs()
            f = torch.exp(-self.nu * tau * self.k2) if self.visc_if else None
            for c in range(3):
                self.g[c].mul_(a).add_(r[c])
                self.u[c].add_(self.g[c], alpha=b)
                if f is not None:
                    self.g[c].mul_(f)
                    self.u[c].mul_(f)
            self.project(self.u)

    def velocity(self):
        return torch.stack([self.real(c) for c in self.u])

    def vmax(self):
        return math.sqrt(float(sum(self.real(c).square() for c in self.u).max()))

    def row(self):
        v = [self.real(c) for c in self.u]
        w = [self.real(c) for c in self.vorticity_hat()]
        e = float(sum(c.square().mean() for c in v)) / 2
        z = float(sum(c.square().mean() for c in w)) / 2
        return [e, 2.0 * self.nu * z, z, self.vmax()]


def box_field(case, seed):
    """A smooth random velocity on the box, its spectrum in the full layout [z][y][x]."""
    shape = (case["nz"], case["ny"], case["nx"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, k2, keep, _ = box_modes(case)
    decay = torch.exp(-k2 / (0.02 * k2.max()))
    u = [torch.fft.fftn(torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)) * decay
         for _ in range(3)]
    box_project(u, k, k2, keep)
    rms = math.sqrt(float(sum(torch.fft.ifftn(c).real.square().mean() for c in u)))
    return [c / rms for c in u]


def box_modes(case):
    m, k, half = [], [], 0.0
    for j, (n, length) in enumerate(((case["nx"], case["lx"]), (case["ny"], case["ly"]), (case["nz"], case["lz"]))):
        i = torch.arange(n, dtype=torch.float64, device="cuda")
        shape = [1, 1, 1]
        shape[2 - j] = n
        m.append((torch.where(i <= n // 2, i, i - n).square() / (n / 2.0) ** 2).view(shape))
        k.append((TWO_PI / length * torch.where(i <= n // 2, i, i - n)).view(shape))
        half = half + k[j] * (0.5 * length / n)
    keep = m[0] + m[1] + m[2] <= 1.0
    return k, k[0] * k[0] + k[1] * k[1] + k[2] * k[2], keep, torch.polar(torch.ones_like(half), half)


def box_project(f, k, k2, keep):
    dot = (f[0] * k[0] + f[1] * k[1] + f[2] * k[2]) / torch.where(k2 > 0, k2, torch.ones_like(k2))
    for c in range(3):
        f[c].sub_(dot * k[c]).mul_(keep & (k2 > 0))


def box_exact(case, seed):
    k, k2, keep, phase = box_modes(case)
    u = box_field(case, seed)
    g = [torch.zeros_like(c) for c in u]
    dt = 0.05 * min(case["lx"] / case["nx"], case["ly"] / case["ny"], case["lz"] / case["nz"])
    for _ in range(case["steps"]):
        for a, b in ((0.0, dt / 3.0), (-5.0 / 9.0, 15.0 * dt / 16.0), (-153.0 / 128.0, 8.0 * dt / 15.0)):
            v = [torch.fft.ifftn(c).real for c in u]
            vs = [torch.fft.ifftn(c * phase).real for c in u]
            r = [torch.zeros_like(c) for c in u]
            for i in range(3):
                for j in range(i, 3):
                    p = torch.fft.fftn(v[i] * v[j])
                    if case["dealias"]:
                        p = 0.5 * (p + torch.fft.fftn(vs[i] * vs[j]) * phase.conj())
                    p = p * keep * -1j
                    r[i] += p * k[j]
                    if i != j:
                        r[j] += p * k[i]
            r = [r[c] - 1e-3 * k2 * u[c] for c in range(3)]
            box_project(r, k, k2, keep)
            for c in range(3):
                g[c] = a * g[c] + r[c]
                u[c] = u[c] + b * g[c]
            box_project(u, k, k2, keep)
    return [c.cpu().numpy() for c in u]


def exact(case, seed):
    kind = case["kind"]
    if kind == "forward":
        return torch.fft.fftn(prepare(case, seed)["phys"])
    if kind == "box":
        return box_exact(case, seed)
    if kind == "solve":
        n, dx = case["n"], TWO_PI / case["n"]
        o = Exact(n, 1.0 / case["re"], seed, case.get("visc_if", False), case.get("rotational", False))
        for _ in range(case["steps"]):
            o.step(dt_of(n) if case["stepping"] == "fixed" else min(0.5, CFL * dx / o.vmax()))
        out = dict(velocity=o.velocity().cpu())
        if case["stepping"] == "loop":
            out["row"] = o.row()
        return out
    out = []
    for sp in members(case, seed):
        o = Exact(sp["n"], sp["nu"], sp["seed"])
        dx = TWO_PI / sp["n"]
        if kind == "ensemble":
            for _ in range(case["steps"]):
                o.step(min(0.5, CFL * dx / o.vmax()))
            out.append(o.velocity().cpu())
        else:
            t, steps = 0.0, 0
            while t < case["t_end"] - 1e-14:
                dt = min(min(0.5, CFL * dx / o.vmax()), case["t_end"] - t)
                o.step(dt)
                t, steps = t + dt, steps + 1
            out.append(dict(steps=steps, row=np.array(o.row())))
    return out

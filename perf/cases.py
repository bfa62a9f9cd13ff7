"""The workloads on which this framework's speed is measured, and their values in 64 bits.

A case is a set of half-channel LES instances that a program advances by a
few time steps and then looks at: ``prepare`` makes the handles and takes
them past their special first steps, ``run`` advances all of them and reads
velocity and pressure back into page-locked host memory, as a program does
that analyses or stores the flow every few steps.  Keys of a case:

  grids      "NXxNYxNZ:COUNT,...": the grid classes and their instances.  One
             instance alone is a LesgoGPU, several (or several classes, whose
             steps overlap on the device) are one LesgoBatch per class
  precision  "mixed", "fp64" or "fp64dw"
  form       "fused": step(); "dropin": the stage entry points in the
             reference's order (single instances)
  steps      time steps per pass, a multiple of the dynamic model's five
  disks      actuator disks per instance, in rows of four
  cfl        0: fixed time step; else the CFL number it is chosen from

Results of the mixed form are kept in single precision, the others in double.
"""
import math

import numpy as np
import torch

from lesgo_gb300.solver import LesgoBatch, LesgoGPU

LX, LY, LZ = 2.0 * math.pi, math.pi, 1.0
ZI, USTAR, VONK = 1000.0, 0.45, 0.4
CS_COUNT = 5
SPIN_UP = 5          # past the Euler step and the start of the dynamic model


def _case(name, grids, precision="mixed", form="fused", steps=5, disks=0, cfl=0.0):
    return dict(name=name, grids=grids, precision=precision, form=form, steps=steps, disks=disks, cfl=cfl)


def listed():
    return [
        # the smallest calls: one small instance, where launches and latency count
        _case("fp64-32", "32x32x32:1", "fp64", steps=10),
        _case("mixed-48", "48x48x48:1", steps=10),
        # a solver that calls the stages one by one, as the Fortran main loop does
        _case("dropin-fp64-64", "64x64x64:1", "fp64", "dropin"),
        _case("dropin-mixed-96", "96x96x64:1", "mixed", "dropin"),
        # an uneven grid with factors of three, and an odd number of levels
        _case("mixed-192x96x41", "192x96x41:1"),
        # the 128^3 half channel in each precision form
        _case("mixed-128", "128x128x128:1"),
        _case("fp64-128", "128x128x128:1", "fp64"),
        _case("fp64dw-128", "128x128x128:1", "fp64dw"),
        # a served chunk: a few instances of one ragged grid
        _case("batch6-108x72x30", "108x72x30:6"),
        # the ensemble of uneven grids that the benchmark reports
        _case("ensemble-48", "48x48x48:15,64x64x64:13,96x96x64:9,128x64x64:11"),
        # the largest: the wind farm, its time step chosen from the CFL number
        _case("windfarm-256x256x192", "256x256x192:1", disks=12, cfl=0.0625),
    ]


# most grid points of a drawn case, by precision (a pass costs less than the largest listed one)
_MOST = {"mixed": 8_000_000, "fp64": 1_500_000, "fp64dw": 2_500_000}
_NX = (32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256)
_NY = (24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 256)


def draw(rng):
    precision = rng.choice(("mixed", "mixed", "mixed", "mixed", "fp64", "fp64dw"))
    form = rng.choice(("fused", "fused", "fused", "dropin"))
    classes = 1 if form == "dropin" else rng.choice((1, 1, 1, 2, 3))
    grids = []
    for _ in range(classes):
        while True:
            nx, ny = rng.choice(_NX), rng.choice(_NY)
            nz = round(math.exp(rng.uniform(math.log(12), math.log(192))))
            room = _MOST[precision] // classes // (nx * ny * nz)
            if room >= 1 and nx <= 4 * ny and ny <= 2 * nx:
                break
        most = 1 if form == "dropin" else min(room, 16)
        grids.append("%dx%dx%d:%d" % (nx, ny, nz, round(math.exp(rng.uniform(0, math.log(most))))))
    c = _case("", ",".join(grids), precision, form)
    if form == "fused" and classes == 1 and rng.random() < 0.2:
        c["disks"], c["cfl"] = rng.choice((1, 4, 12)), 0.05
    del c["name"]
    return c


def _classes(case):
    for part in case["grids"].split(","):
        grid, count = part.split(":")
        yield tuple(int(n) for n in grid.split("x")), int(count)


def _instances(case, seed):
    """(class, nx, ny, Nz, [(zo, seed of the initial condition), ...])"""
    rng = np.random.RandomState(seed % (1 << 31))
    for c, ((nx, ny, nz), count) in enumerate(_classes(case)):
        yield c, nx, ny, nz, [(10.0 ** rng.uniform(-5, -3), int(rng.randint(1, 1 << 30))) for _ in range(count)]


def _dt(nx):
    return 2.0e-4 * min(1.0, 128.0 / nx)    # below an advective CFL number of about 0.1


def _disks(case):
    """Disks of diameter 0.1 at hub height 0.1, seven diameters apart along the flow and five across."""
    return [dict(xloc=1.0 + 0.7 * (i % 4), yloc=1.0 + 0.5 * (i // 4), height=0.1, dia=0.1, thk=0.0, theta1=0.0,
                 theta2=0.0, Ct_prime=1.33) for i in range(case["disks"])]


FIELDS = ("u", "v", "w", "p")


def prepare(case, seed):
    single = torch.float32 if case["precision"] == "mixed" else None
    groups = []
    for _, nx, ny, nz, insts in _instances(case, seed):
        kw = dict(nx=nx, ny=ny, Nz=nz, dt=_dt(nx), dyn_init=CS_COUNT, cs_count=CS_COUNT, precision=case["precision"])
        if case["cfl"]:
            kw.update(use_cfl_dt=True, cfl=case["cfl"])
        if len(insts) == 1 and "," not in case["grids"]:
            zo, ic = insts[0]
            h, ids = LesgoGPU(zo=zo, turbines=_disks(case), **kw), [None]
            h.init_ic(ic)
        else:
            h = LesgoBatch(len(insts), **kw)
            ids = [h.add(zo, ic, _disks(case)) for zo, ic in insts]
        host = torch.empty((len(ids), 4, nz + 2, ny, nx + 2), dtype=torch.float64, pin_memory=torch.cuda.is_available())
        view = host[:, :, 1:, :, :nx]       # levels 1..nz, without the row padding
        flow = torch.empty(view.shape, dtype=single) if single else view
        groups.append((h, ids, host, view, flow))
    for h, *_ in groups:
        h.step(SPIN_UP)
    state = dict(steps=case["steps"], dropin=case["form"] == "dropin", disks=case["disks"], single=single, groups=groups)
    for h, *_ in groups:
        h.sync()
    return state


def run(state):
    for h, *_ in state["groups"]:
        if state["dropin"]:
            for _ in range(state["steps"]):
                h.step_reference_order()
        else:
            h.step(state["steps"])
    for h, ids, host, _, _ in state["groups"]:
        last = host.shape[2] - 1
        for n, iid in enumerate(ids):
            for f, name in enumerate(FIELDS):
                where = host[n, f].data_ptr()
                if iid is None:
                    h.get_ptr(name, where, 0, last, wait=False)
                else:
                    h.get_ptr(iid, name, where, 0, last, wait=False)
    out = []
    for h, ids, _, view, flow in state["groups"]:
        h.sync()
        if flow is not view:
            flow.copy_(view)
        out.append(dict(velocity=flow[:, :3], pressure=flow[:, 3]))
    if state["disks"]:
        h, ids = state["groups"][0][:2]
        power = np.stack([(h.turbine_state() if i is None else h.turbine_state(i))["power"] for i in ids])
        out.append(dict(power=power.astype(np.float32) if state["single"] else power))
    return out


def work(case):
    """A step reads and writes the velocity, its right-hand sides and the model coefficient, one step in five the four
    running averages too; a pass writes velocity and pressure for the host.  The transforms of a step: 17 to spectra
    and 16 back (with the pressure's), 6 back and 3 forward on the 3/2 grid, and in one step of five 21 and 42."""
    size = 4 if case["precision"] == "mixed" else 8
    nbytes = flops = 0.0
    for (nx, ny, nz), count in _classes(case):
        n = nx * ny * nz * count
        nbytes += n * (case["steps"] * (14 + 8 / CS_COUNT) * size + 4 * 8)
        plane = 2.5 * nx * ny * math.log2(nx * ny)
        big = 2.5 * 2.25 * nx * ny * math.log2(2.25 * nx * ny)
        flops += case["steps"] * count * nz * (plane * (17 + 16 + 63 / CS_COUNT) + big * 9 + 250.0 * nx * ny)
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------------
# The same time steps in 64 bits, in plain torch
# --------------------------------------------------------------------------
def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out, power = [], []
    for _, nx, ny, nz, insts in _instances(case, seed):
        flows = []
        for zo, ic in insts:
            s = _Channel(nx, ny, nz, zo, ic, _dt(nx), _disks(case), case["cfl"], dev)
            for _ in range(SPIN_UP + case["steps"]):
                s.step()
            flows.append(torch.stack([s.u[1:], s.v[1:], s.w[1:], s.p[1:]]).cpu())
            power.append([d["power"] for d in s.disks])
        flow = torch.stack(flows)
        out.append(dict(velocity=flow[:, :3], pressure=flow[:, 3]))
    if case["disks"]:
        out.append(dict(power=np.array(power)))
    return out


def _signed(c):
    return c - (1 << 64) if c >= 1 << 63 else c


def _shift(x, n):
    return (x >> n) & ((1 << (64 - n)) - 1)


def _noise(seed, field, k, j, i):
    """U(-1, 1) from the splitmix64 hash of (seed, field, level, row, column), zero-based."""
    x = (((seed * 8 + field) * 65536 + k) * 65536 + j) * 65536 + i + _signed(0x9E3779B97F4A7C15)
    x = (x ^ _shift(x, 30)) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ _shift(x, 27)) * _signed(0x94D049BB133111EB)
    x = x ^ _shift(x, 31)
    return 2.0 * (_shift(x, 11).double() * 2.0 ** -53) - 1.0


class _Channel:
    """One half channel: log-law wall below, stress-free lid above, spectral in x and y, staggered in z.  Arrays are
    (level 0..nz, y, x); u, v, p and their like stand at cell middles, w and its like at cell faces."""

    def __init__(self, nx, ny, nz, zo, ic, dt, disks, cfl, dev):
        self.nx, self.ny, self.nz, self.zo, self.dev = nx, ny, nz + 1, zo, dev
        nz = self.nz
        self.dx, self.dy, self.dz = LX / nx, LY / ny, LZ / (nz - 1)
        self.dt, self.cfl, self.t1, self.t2 = dt, cfl, 1.5, -0.5
        self.ldt = 0.0 if cfl else CS_COUNT * dt
        self.delta = (self.dx * self.dy * self.dz) ** (1.0 / 3.0)
        real = dict(dtype=torch.float64, device=dev)
        mx, my = torch.arange(nx // 2 + 1, **real), torch.fft.fftfreq(ny, 1.0 / ny, **real)
        self.keep = torch.ones((ny, nx // 2 + 1), **real)
        self.keep[ny // 2] = 0.0
        self.keep[:, -1] = 0.0
        self.kx = 2 * math.pi / LX * mx[None, :] * self.keep
        self.ky = 2 * math.pi / LY * my[:, None] * self.keep
        k2 = self.kx ** 2 + self.ky ** 2
        self.G = [torch.where(k2 >= (math.pi / (a * math.sqrt(self.dx * self.dy))) ** 2, 0.0, self.keep) for a in (2.0, 4.0)]
        k, j, i = (torch.arange(n, dtype=torch.int64, device=dev) for n in (nz, ny, nx))
        k, j, i = k[1:, None, None], j[None, :, None], i[None, None, :]
        z = (torch.arange(1, nz, **real) - 0.5) * self.dz
        full = lambda: torch.zeros((nz + 1, ny, nx), **real)  # noqa: E731
        self.u, self.v, self.w, self.p, self.cs = full(), full(), full(), full(), full()
        self.rhs = [full() for _ in range(3)]
        self.u[1:nz] = 2.5 * torch.log(z / zo)[:, None, None] * (1.0 + 0.1 * _noise(ic, 0, k, j, i))
        self.v[1:nz] = 0.1 * _noise(ic, 1, k, j, i)
        self.w[1:nz] = 0.1 * _noise(ic, 2, k, j, i)
        self.w[1] = 0.0
        self.u[nz], self.v[nz] = self.u[nz - 1], self.v[nz - 1]
        self.avg, self.jt = None, 0
        self.disks = [self._disk(**d) for d in disks]

    # ---- spectral operators ----
    def _fwd(self, f):
        return torch.fft.rfft2(f) * self.keep

    def _inv(self, F):
        return torch.fft.irfft2(F, s=(self.ny, self.nx))

    def _big(self, f):
        """to the 3/2 grid"""
        ny, h, m = self.ny, self.ny // 2, self.nx // 2
        F = self._fwd(f)
        B = torch.zeros(f.shape[:-2] + (3 * ny // 2, 3 * self.nx // 4 + 1), dtype=F.dtype, device=self.dev)
        B[..., :h, :m] = F[..., :h, :m]
        B[..., 3 * ny // 2 - h + 1:, :m] = F[..., h + 1:, :m]
        return torch.fft.irfft2(B, s=(3 * ny // 2, 3 * self.nx // 2)) * 2.25

    def _small(self, f):
        """back from it"""
        ny, h, m = self.ny, self.ny // 2, self.nx // 2
        B = torch.fft.rfft2(f)
        F = torch.zeros(f.shape[:-2] + (ny, m + 1), dtype=B.dtype, device=self.dev)
        F[..., :h, :m] = B[..., :h, :m]
        F[..., h + 1:, :m] = B[..., 3 * ny // 2 - h + 1:, :m]
        return torch.fft.irfft2(F, s=(ny, self.nx)) / 2.25

    def _test(self, f, n):
        return self._inv(torch.fft.rfft2(f) * self.G[n])

    # ---- one time step ----
    def step(self):
        nz, dz = self.nz, self.dz
        if self.cfl:
            before = self.dt
            m = [float(a[1:nz].abs().max()) / d for a, d in ((self.u, self.dx), (self.v, self.dy), (self.w, dz))]
            self.dt = self.cfl / max(m)
            self.t1 = 1.0 + 0.5 * self.dt / before
            self.t2 = 1.0 - self.t1
            self.ldt += self.dt
        self.jt += 1
        old = self.rhs
        grad = []
        for a in (self.u, self.v, self.w):
            F = self._fwd(a[1:])
            a[1:] = self._inv(F)
            for k in (self.kx, self.ky):
                g = torch.zeros_like(a)
                g[1:] = self._inv(1j * k * F)
                grad.append(g)
        ux, uy, vx, vy, wx, wy = grad
        uz, vz, wz = (torch.zeros_like(ux) for _ in range(3))
        uz[2:nz] = (self.u[2:nz] - self.u[1:nz - 1]) / dz
        vz[2:nz] = (self.v[2:nz] - self.v[1:nz - 1]) / dz
        wz[1:nz] = (self.w[2:] - self.w[1:nz]) / dz
        # the wall: log law on the filtered velocity
        uf, vf = self._test(self.u[1], 0), self._test(self.v[1], 0)
        speed = torch.sqrt(uf ** 2 + vf ** 2)
        ustar = speed * VONK / math.log(0.5 * dz / self.zo)
        wall = -ustar ** 2 / speed * uf, -ustar ** 2 / speed * vf
        uz[1] = ustar / (0.5 * dz * VONK) * self.u[1] / speed
        vz[1] = ustar / (0.5 * dz * VONK) * self.v[1] / speed
        tau = self._stress(ux, uy, uz, vx, vy, vz, wx, wy, wz, wall)
        div = self._divergence(*tau)
        conv = self._convection(uy, uz, vx, vz, wx, wy)
        force = self._forces()
        new = [-c - d + f for c, d, f in zip(conv, div, force)]
        new[0][1:nz] += 1.0 / LZ            # the mean pressure gradient
        if self.jt == 1:
            old = new
        for n, a in enumerate((self.u, self.v, self.w)):
            top = nz + 1 if n == 2 else nz
            a[1:top] += self.dt * (self.t1 * new[n][1:top] + self.t2 * old[n][1:top])
        px, py, pz = self._pressure(div[2])
        for a, r, g, lo in ((self.u, new[0], px, 1), (self.v, new[1], py, 1), (self.w, new[2], pz, 2)):
            r -= g
            a[lo:nz] -= self.dt * self.t1 * g[lo:nz]
        self.u[nz], self.v[nz] = self.u[nz - 1], self.v[nz - 1]
        self.w[nz] = 0.0
        self.w[1] = 0.0
        self.rhs = new

    def _stress(self, ux, uy, uz, vx, vy, vz, wx, wy, wz, wall):
        nz = self.nz
        S = [torch.zeros_like(ux) for _ in range(6)]      # 11 12 13 22 23 33 at cell faces
        c, m = slice(2, nz), slice(1, nz - 1)
        for n, (a, b) in enumerate(((ux, ux), (uy, vx), (None, None), (vy, vy), (None, None), (wz, wz))):
            if a is not None:
                S[n][c] = 0.25 * (a[c] + a[m] + b[c] + b[m])
                S[n][1] = 0.5 * (a[1] + b[1])
                S[n][nz] = 0.5 * (a[nz - 1] + b[nz - 1])
        S[5][nz] = 0.5 * wz[nz - 1]
        for n, a, b in ((2, uz, wx), (4, vz, wy)):
            S[n][2:] = 0.5 * (a[2:] + b[2:])
            S[n][1] = 0.5 * (a[1] + 0.5 * (b[1] + b[2]))
        if self.jt == 1:
            self.cs[:] = 0.03
        elif self.jt >= CS_COUNT and self.jt % CS_COUNT == 0:
            self._dynamic(S)
        nu = _magnitude(S) * self.cs * self.delta ** 2
        t = [torch.zeros_like(ux) for _ in range(6)]
        for n in (0, 1, 3, 5):
            t[n][2:nz] = -0.5 * (nu[2:nz] + nu[3:]) * (S[n][2:nz] + S[n][3:])
            t[n][1] = -2.0 * nu[1] * S[n][1]
        for n in (2, 4):
            t[n][2:nz] = -2.0 * nu[2:nz] * S[n][2:nz]
            t[n][1] = wall[n // 2 - 1]
        return t

    def _dynamic(self, S):
        """The Lagrangian scale-dependent model: the coefficient at cell faces from test filters at two scales."""
        nz, ldt, tiny = self.nz, self.ldt, 1.0e-24
        u, v, w = (torch.zeros_like(self.u) for _ in range(3))
        u[2:nz], v[2:nz] = 0.5 * (self.u[2:nz] + self.u[1:nz - 1]), 0.5 * (self.v[2:nz] + self.v[1:nz - 1])
        w[2:nz] = self.w[2:nz]
        u[1], v[1], w[1] = self.u[1], self.v[1], 0.25 * self.w[2]
        u[nz], v[nz] = self.u[nz - 1], self.v[nz - 1]
        vel, Sm = (u[1:], v[1:], w[1:]), _magnitude(S)
        pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
        new = []
        for n, a in ((0, 2.0), (1, 4.0)):
            bar = [self._test(x, n) for x in vel]
            L = [self._test(vel[i] * vel[j], n) - bar[i] * bar[j] for i, j in pairs]
            Sb = [self._test(x[1:], n) for x in S]
            Sbm = _magnitude(Sb)
            M = [2 * self.delta ** 2 * (self._test((Sm * x)[1:], n) - a * a * Sbm * y) for x, y in zip(S, Sb)]
            new += [_contract(L, M), _contract(M, M)]
        if self.avg is None:
            self.avg = [0.03 * new[1], new[1], 0.03 * new[3], new[3]]
        else:
            self.avg = self._transported(u, v, w)
        cs = []
        for n in (0, 2):
            a, b = self.avg[n], self.avg[n + 1]
            T = 1.5 * self.delta * torch.clamp(a * b, min=tiny) ** -0.125
            e = ldt / T
            e = e / (1.0 + e)
            a = torch.clamp(e * new[n] + (1.0 - e) * a, min=tiny)
            b = e * new[n + 1] + (1.0 - e) * b
            self.avg[n], self.avg[n + 1] = a, b
            cs.append(torch.clamp(a / (b + tiny), min=tiny))
        beta = cs[1] / cs[0]
        beta[nz - 1] = 1.0
        self.cs[1:] = torch.clamp(cs[0] / torch.clamp(beta, min=0.125), min=tiny)
        if self.cfl:
            self.ldt = 0.0

    def _transported(self, u, v, w):
        """The running averages at the points from which the flow has come."""
        nz, dz = self.nz, self.dz
        k, j, i = (torch.arange(n, dtype=torch.float64, device=self.dev) for n in (nz, self.ny, self.nx))
        x = torch.remainder(i[None, None, :] - u[1:] * self.ldt / self.dx, self.nx)
        y = torch.remainder(j[None, :, None] - v[1:] * self.ldt / self.dy, self.ny)
        z = k[:, None, None] - w[1:] * self.ldt / dz
        z[0] += 0.5                              # the first level stands half a cell above the wall
        i0, j0, k0 = x.floor().long(), y.floor().long(), torch.clamp(z.floor().long(), 0, nz - 2)
        fx, fy, fz = x - i0, y - j0, z - k0
        low = z < 1.0                            # between the first two levels, half a cell apart
        fz = torch.where(low, torch.clamp(2.0 * (z - 0.5), min=0.0), fz)
        i0, j0 = i0 % self.nx, j0 % self.ny
        i1, j1, k1 = (i0 + 1) % self.nx, (j0 + 1) % self.ny, k0 + 1
        out = []
        for F in self.avg:
            at = lambda K: (F[K, j0, i0] * (1 - fx) + F[K, j0, i1] * fx) * (1 - fy) + (F[K, j1, i0] * (1 - fx) + F[K, j1, i1] * fx) * fy  # noqa: E731
            out.append(at(k0) * (1 - fz) + at(k1) * fz)
        return out

    def _divergence(self, t11, t12, t13, t22, t23, t33):
        nz, dz = self.nz, self.dz
        out = []
        for a, b, c, uv in ((t11, t12, t13, True), (t12, t22, t23, True), (t13, t23, t33, False)):
            d = torch.zeros_like(a)
            d[1:] = self._inv(1j * self.kx * self._fwd(a[1:]) + 1j * self.ky * self._fwd(b[1:]))
            if uv:
                d[1:nz] += (c[2:] - c[1:nz]) / dz
                d[nz] = 0.0
            else:
                d[2:nz] += (c[2:nz] - c[1:nz - 1]) / dz
            out.append(d)
        return out

    def _convection(self, uy, uz, vx, vz, wx, wy):
        nz = self.nz
        o1, o2 = wy - vz, uz - wx
        o1[1] = 0.5 * (wy[1] + wy[2]) - vz[1]
        o2[1] = uz[1] - 0.5 * (wx[1] + wx[2])
        u, v, w, o1, o2, o3 = (self._big(a[1:]) for a in (self.u, self.v, self.w, o1, o2, vx - uy))
        n = nz - 1                                        # here entry 0 is level 1
        cx, cy, cz = (torch.zeros_like(u) for _ in range(3))
        a, b = w * o2, -w * o1
        for c, f, vort in ((cx, a, -v * o3), (cy, b, u * o3)):
            c[:n] = vort[:n]
            c[1:n - 1] += 0.5 * (f[2:n] + f[1:n - 1])
            c[0] += 0.5 * f[1]
            c[n - 1] += 0.5 * f[n - 1]
        cz[1:n] = 0.5 * ((v[1:n] + v[:n - 1]) * o1[1:n] - (u[1:n] + u[:n - 1]) * o2[1:n])
        out = []
        for c in (cx, cy, cz):
            r = torch.zeros_like(self.u)
            r[1:] = self._small(c)
            out.append(r)
        return out

    def _pressure(self, divtz):
        nz, dz, ny, nx = self.nz, self.dz, self.ny, self.nx
        Hx, Hy, Hz = (self._fwd(a / (self.t1 * self.dt)) for a in (self.u, self.v, self.w))
        low, top = self._fwd(divtz[1]), self._fwd(divtz[nz])
        r = torch.zeros((nz + 1,) + low.shape, dtype=low.dtype, device=self.dev)
        r[0], r[nz] = -dz * low, -dz * top
        r[1:nz] = 1j * self.kx * Hx[1:nz] + 1j * self.ky * Hy[1:nz] + (Hz[2:] - Hz[1:nz]) / dz
        c, mid = 1.0 / dz ** 2, -(self.kx ** 2 + self.ky ** 2 + 2.0 / dz ** 2)
        skip = (self.kx == 0) & (self.ky == 0)            # the mean mode and the unused ones
        r *= torch.where(skip, 0.0, 1.0)
        bet = -torch.ones_like(mid)
        ph, gam = torch.zeros_like(r), torch.zeros((nz + 1,) + mid.shape, dtype=mid.dtype, device=self.dev)
        ph[0] = r[0] / bet
        for j in range(1, nz + 1):
            a, b, above = (c, mid, c if j > 1 else 1.0) if j < nz else (-1.0, torch.ones_like(mid), c)
            gam[j] = above / bet
            bet = torch.where(skip, torch.ones_like(mid), b - a * gam[j])
            ph[j] = (r[j] - a * ph[j - 1]) / bet
        for j in range(nz - 1, -1, -1):
            ph[j] -= gam[j + 1] * ph[j + 1]
        ph[1, 0, 0] = -dz * low[0, 0]
        ph[2:, 0, 0] = ph[1, 0, 0] + torch.cumsum(Hz[2:, 0, 0] * dz, 0)
        self.p = self._inv(ph)
        px, py, pz = (torch.zeros_like(self.p) for _ in range(3))
        px[1:nz], py[1:nz] = self._inv(1j * self.kx * ph[1:nz]), self._inv(1j * self.ky * ph[1:nz])
        pz[1:] = (self.p[1:] - self.p[:nz]) / dz
        return px, py, pz

    # ---- actuator disks ----
    def _disk(self, xloc, yloc, height, dia, thk, theta1, theta2, Ct_prime):
        """The points a disk facing the flow acts on and their weights: the disk smeared by a Gaussian."""
        dx, dy, dz, nx, ny = self.dx, self.dy, self.dz, self.nx, self.ny
        thk = max(thk, dx * float(np.float32(1.01)))
        width = 1.5 * math.sqrt(dx * dx + dy * dy + dz * dz)
        half, s = 0.5 * dia, width / (0.5 * dia)
        N, L = 2048, 1 + 10 * s / math.sqrt(12.0)
        d = 2 * L / N
        yz = -L + d * (np.arange(1, N + 1) - 0.5)
        r2 = yz[:, None] ** 2 + yz[None, :] ** 2
        g = 6.0 / (math.pi * s ** 2) * np.exp(-6 * r2 / s ** 2)
        h = np.where(np.sqrt(r2) < 1, 1.0 / math.pi, 0.0)
        R = np.fft.irfft2(np.fft.rfft2(g) * np.fft.rfft2(h) * d ** 2, s=(N, N))[:N // 2, 0]
        r = yz[:N // 2] + L
        R = R / np.sum(2 * math.pi * r * R * d)
        M = float(np.sum(2 * math.pi * r * R ** 2 * d) * math.pi)
        erf = np.vectorize(math.erf)

        def weight(rad, ax):
            ax, b = ax / half, 0.5 * thk / half
            e = math.sqrt(6.0) / s
            return 0.5 / (2 * b) * (erf(e * (ax + b)) - erf(e * (ax - b))) * np.interp(rad / half, r, R) / half ** 3

        reach = 0.5 * dia + 3 * width
        near = lambda q: int(math.floor(q + 0.5))  # noqa: E731
        ic, jc, kc = near(xloc / dx), near(yloc / dy), near(height / dz + 0.5)
        im, jm = min(int(reach / dx + 2), nx // 2), min(int(reach / dy + 2), ny // 2)
        k, j, i = np.meshgrid(np.arange(1, self.nz + 1), np.arange(jc - jm, jc + jm), np.arange(ic - im, ic + im), indexing="ij")
        rx, ry, rz = i * dx - xloc, j * dy - yloc, (k - 0.5) * dz - height
        ind = weight(np.sqrt(ry * ry + rz * rz), np.abs(rx))
        pick = ind > 1e-2 * float(weight(np.zeros(1), np.zeros(1))[0])
        ind = ind[pick] / np.sum(ind[pick] * dx * dy * dz)
        at = tuple(torch.from_numpy(q[pick] % n if n else q[pick]).to(self.dev) for q, n in ((k, 0), (j, ny), (i, nx)))
        return dict(at=at, ind=torch.from_numpy(ind).to(self.dev), M=M, dia=dia, ct=Ct_prime, power=0.0)

    def _forces(self):
        """An actuator disk facing the flow pushes along x only."""
        f = [torch.zeros_like(self.u) for _ in range(3)]
        thrust = []
        for d in self.disks:
            v = -float((self.u[d["at"]] * d["ind"]).sum()) * self.dx * self.dy * self.dz
            v /= 1 + 0.25 * (1 - d["M"]) * d["ct"]
            t = -0.5 * d["ct"] * abs(v) * v * 0.25 * math.pi * d["dia"] ** 2
            d["power"] = -t * v
            thrust.append(t)
        for d, t in zip(self.disks, thrust):     # where disks meet, the last one acts
            f[0][d["at"]] = -t * d["ind"]
        return f


def _magnitude(S):
    return torch.sqrt(2.0 * (S[0] ** 2 + S[3] ** 2 + S[5] ** 2 + 2.0 * (S[1] ** 2 + S[2] ** 2 + S[4] ** 2)))


def _contract(A, B):
    return A[0] * B[0] + A[3] * B[3] + A[5] * B[5] + 2.0 * (A[1] * B[1] + A[2] * B[2] + A[4] * B[4])

"""Performance cases of the framework: RK3 steps of the lomacte mixing layer
over the range of grids, precision forms and options that its runs use.

A case names the grids that are resident together ("256x257x256", several
of them separated by commas for an ensemble), the precision form, the
options of the run and how many RK3 steps one pass advances.  ``prepare``
makes the seeded initial condition, creates the handles and loads them;
``run`` advances every resident case and returns its updated state.

The FP64 form returns the state fields where they are (views of the device
memory, layout [y][kx][kz]).  The mixed forms return them in single
precision, the type a run's images and restart files store them in; their
last digits beyond that are not results of a mixed run.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from loma_phd_b200 import lomacte as L

CFL, NCFL = 0.5, 10  # Deltat from CFL = 0.5 every 10 steps (dt = 0 in a case)
PR = float(np.float32(0.7))  # Pr = Sc
SIGMA = 0.7  # mu = T^0.7
FIELDS = ("vor", "phi", "psi", "scal")
DIAG = ("time", "Deltat", "dm", "dw", "Redw", "trapz", "masst", "massu", "massv", "massw", "H00u", "H00w",
        "Deltat_next")

# nx and nz the library transforms (2/3 of a transform length)
MODES = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768)


def _case(name, grids, form, steps, **kw):
    c = dict(name=name, grids=grids, form=form, steps=steps, scalar=False, visc=False, Re=160.0, s=4.0, dt=0.01,
             monitor=False, stats=False)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest grid of the test suite, one step per call: latency
        _case("latency_24_fp64", "24x33x24", 0, 1),
        # the small plain run (64 modes, ny = 129, mu = T^0.7 and the
        # scalar), FP64, with its diagnostics and the scalar read back
        _case("small_64_fp64_mu_z", "64x129x64", 0, 4, scalar=True, visc=True, monitor=True),
        # one request of the serving stream: 3-D, constant viscosity, the
        # CFL mode, in the server's chunks of eight steps
        _case("serve_96_mixed", "96x129x96", 1, 8, Re=400.0, s=2.5, dt=0.0),
        # a 2-D request of the stream (one kz mode)
        _case("serve_2d_512_fp64", "512x257x1", 0, 8, Re=300.0, s=3.0, dt=0.0),
        # requests of uneven grids resident together, one stream each
        _case("serve_6_uneven_mixed", "64x97x64,128x129x96,96x193x128,64x129x64,192x97x64,256x257x1", 1, 8, Re=250.0,
              s=3.0, dt=0.0),
        # the largest grid of the ensemble, FP64, nx != nz
        _case("ensemble_192_fp64", "192x193x128", 0, 2, Re=300.0, s=3.0),
        # a run that accumulates statistics on every step
        _case("stats_128_fp64", "128x129x128", 0, 2, stats=True),
        # the medium run, both forms
        _case("medium_256_fp64_mu_z", "256x257x256", 0, 2, scalar=True, visc=True, monitor=True),
        _case("medium_256_mixed_mu_z", "256x257x256", 1, 2, scalar=True, visc=True, monitor=True),
        # the large run's transform lengths (1152 points) at a ny of which
        # three fit the card, both forms, and the more exact mixed form
        _case("large_768_fp64_mu_z", "768x33x768", 0, 2, scalar=True, visc=True, Re=800.0, s=8.0, dt=0.0,
              monitor=True),
        _case("large_768_mixed_mu_z", "768x65x768", 1, 2, scalar=True, visc=True, Re=800.0, s=8.0, dt=0.0,
              monitor=True),
        _case("large_384_mixed2", "384x129x384", 2, 1, Re=400.0, s=4.0),
    ]


def _sizes(grid):
    nx, ny, nz = (int(v) for v in grid.split("x"))
    return nx, ny, nz


def _cost(case):
    """Grid points times steps, weighted by what the form and the options add."""
    pts = 0
    for gr in case["grids"].split(","):
        nx, ny, nz = _sizes(gr)
        pts += nx * ny * max(nz, 2)
    w = (1.0, 0.7, 1.3)[case["form"]] * (1.3 if case["scalar"] else 1.0) * (1.3 if case["visc"] else 1.0)
    return pts * case["steps"] * w


def draw(rng):
    """A run of the same ranges: nx and nz of any supported size (2-D now
    and then), any ny that the library takes, the three forms, the options."""
    most = max(_cost(c) for c in listed()) / 2
    while True:
        form = rng.choice((0, 0, 1, 1, 1, 2))
        two_d = rng.random() < 0.15
        # form 1 loses phi to FP32 rounding as k^3: short runs at the largest
        # lengths, and 2-D ones (whose |phi| is smaller) up to 256 modes
        nx = rng.choice(((256, 256) if form == 1 else (256, 384, 512, 768)) if two_d else MODES)
        nz = 1 if two_d else rng.choice([m for m in MODES if nx <= 4 * m and m <= 4 * nx])
        ny = int(round(math.exp(rng.uniform(math.log(17), math.log(300)))))
        full = rng.random() < 0.5
        dt = rng.choice((0.0, round(math.exp(rng.uniform(math.log(1e-3), math.log(1e-2))), 5)))
        c = _case("", f"{nx}x{ny}x{nz}", form, rng.randint(1, 2 if form == 1 and max(nx, nz) > 256 else 4), scalar=full or rng.random() < 0.2,
                  visc=full or rng.random() < 0.2, Re=round(rng.uniform(100.0, 400.0), 1),
                  s=round(rng.uniform(1.0, 8.0), 2), dt=dt, stats=form == 0 and rng.random() < 0.2)
        c["monitor"] = c["scalar"] and dt > 0.0
        del c["name"]
        if _cost(c) <= most and L.footprint(_params(c, c["grids"])) > 0:
            return c


def _params(case, grid):
    nx, ny, nz = _sizes(grid)
    fixed = case["dt"] > 0.0
    return L.Params.from_modes(nx, nz, ny, Re=case["Re"], dt_mode=1 if fixed else 0, dt=case["dt"] if fixed else 1e-4,
                               cfl=CFL, ncfl=NCFL, precision=case["form"], scalar=int(case["scalar"]),
                               visc=int(case["visc"]), sigma=SIGMA if case["visc"] else 0.0)


def _initial(case, grid, seed):
    """Parameters, mesh, seeded state and scalar of one resident case."""
    p = _params(case, grid)
    y = L.stretched_mesh(p.my)
    st = L.make_ic(p, y, L.ICParams(s=case["s"], seed=seed))
    z = None
    if case["scalar"]:
        z = np.zeros(p.shape, dtype=np.complex128)
        z[0, 0, :] = 0.5 * (1.0 + np.tanh(y / 2.0))
    return p, y, st, z


def _member_seed(seed, i):
    return (int(seed) * 16 + i) % (1 << 40)


class _DeviceArray:
    """FP64 device memory of a handle, for torch to wrap without a copy."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 2}


def _state_views(g):
    import ctypes
    ptrs = [ctypes.POINTER(ctypes.c_double)() for _ in FIELDS]
    rc = L.lib().lmc_state_device_ptrs(g._h, *[ctypes.byref(q) for q in ptrs])
    if rc != L.LMC_OK:
        raise L.LomacteError(rc, "lmc_state_device_ptrs")
    nkx, mz, my = g.shape
    return [torch.as_tensor(_DeviceArray(ctypes.cast(q, ctypes.c_void_p).value, (my, nkx, mz, 2), g), device="cuda")
            for q in ptrs]


def prepare(case, seed):
    members = []
    for i, grid in enumerate(case["grids"].split(",")):
        p, y, st, z = _initial(case, grid, _member_seed(seed, i))
        g = L.Lomacte(p, y)
        g.load_state(st)
        m = {"g": g, "views": _state_views(g), "stream": torch.cuda.ExternalStream(g.stream)}
        if z is not None:
            g.load_scalar(z)
            m["z"] = torch.empty(p.shape + (2,), dtype=torch.float64, pin_memory=True)
        if case["stats"]:
            g.stats_reset([(p.my + 1) // 2, (p.my + 3) // 4])
        members.append(m)
    return {"case": dict(case), "members": members}


def run(state):
    case = state["case"]
    for m in state["members"]:  # asynchronous, one stream each
        if case["stats"]:
            m["g"].stats_step(case["steps"])
        else:
            m["g"].step(case["steps"])
    if len(state["members"]) > 1:  # the server waits for its chunks before it enqueues the next
        for m in state["members"]:
            m["g"].sync()
    out = []
    for m in state["members"]:
        g = m["g"]
        if case["form"] == 0:
            o = dict(zip(FIELDS, m["views"]))
        else:
            with torch.cuda.stream(m["stream"]):
                o = {k: v.to(torch.float32) for k, v in zip(FIELDS, m["views"])}
        if case["scalar"]:
            g.get_scalar_ptr(m["z"].data_ptr())
            o["Z"] = m["z"]
        if case["monitor"]:
            d = g.diag()
            o["diag"] = np.array([d[k] for k in DIAG], dtype=np.float32 if case["form"] else np.float64)
        if case["stats"]:
            s = g.stats_read()
            o["prof"], o["spec"], o["uner"] = s.prof, s.spec, s.uner
        out.append(o)
    return out


def work(case):
    """Per RK3 substep: the state and its RK3 memory (Omega_y, phi, psi, T,
    the two spectral right-hand sides, RHS(T) in physical space; Z and
    RHS(Z)) read once and written once in FP64; and the operations of the
    transforms (5/2 N log2 N of a real line in x, 5 N log2 N of a complex one
    in z), of the products and of the banded solves along y."""
    nbytes = flops = 0.0
    for grid in case["grids"].split(","):
        p = _params(case, grid)
        sc, vs = int(case["scalar"]), int(case["visc"])
        S = p.nplanes * p.mz * p.my
        P = p.mgalx * p.mgalz * p.my
        fields = 8 + 4 * sc + 6 * vs + 11 + sc
        sub = (6 + sc) * S * 16 * 2 + (1 + sc) * P * 8 * 2
        f = fields * (P * 2.5 * math.log2(p.mgalx) + 5.0 * p.nplanes * p.mgalz * p.my * math.log2(p.mgalz))
        f += P * (50 + 20 * sc + 50 * vs) + S * 2 * (30 * 14 + 30 * 2 * sc + 30 * 3 * vs)
        nbytes += 3 * case["steps"] * sub
        flops += 3 * case["steps"] * f
        if sc:
            nbytes += S * 16
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    out = []
    for i, grid in enumerate(case["grids"].split(",")):
        p, y, st, z = _initial(case, grid, _member_seed(seed, i))
        r = _Plain64(p, y, st, z)
        for n in range(case["steps"]):
            r.step(n % NCFL == 0)
        o = {k: torch.view_as_real(v) for k, v in zip(FIELDS, (r.vor, r.phi, r.psi, r.T))}
        if case["scalar"]:
            o["Z"] = torch.view_as_real(r.Z.permute(1, 2, 0).contiguous())
        if case["monitor"]:
            o["diag"] = np.array([r.diag[k] for k in DIAG])
        if case["stats"]:  # sums over modes: held to the bound of their type
            o["prof"] = o["spec"] = o["uner"] = None
        out.append(o)
    return out


# ----------------------------------------------------------------------
# The same equations in FP64 with torch alone (trunk/lomacte3/src/cross.f:
# 307-1141 and the framework's scalar and viscosity), fields [y][kx][kz].
# ----------------------------------------------------------------------
def _band(rows, offsets, n):
    """Dense matrix from row stencils."""
    A = np.zeros((n, n))
    for j in range(n):
        for c, w in zip(offsets, rows[j]):
            if w != 0.0:
                A[j, j + c] = w
    return A


def _first_derivative(n):
    """Left and right sides of the compact d/deta on [-1, 1] (cfdiff.f:24-182)."""
    h = 2.0 / (n - 1)
    a, b, c = 0.56926818603810, 0.31997939759919, 0.03751544855390
    al = -3 / 4 + 33 / 20 * c + 239 / 180 * a + 82 / 45 * b
    be = 3 / 10 + 24 / 25 * c - 88 / 225 * a + 34 / 225 * b
    de = -1 / 20 + 39 / 100 * c + 19 / 300 * a + 2 / 75 * b
    left = [[de, be, al, 1, al, be, de]] * n
    right = [[-c, -b, -a, 0, a, b, c]] * n
    edge = [([0, 0, 0, 1, 1, 0, 0], [0, 0, 0, -2, 2, 0, 0]),
            ([0, 0, 1 / 4, 1, 1 / 4, 0, 0], [0, 0, -3 / 4, 0, 3 / 4, 0, 0]),
            ([0, 1 / 36, 4 / 9, 1, 4 / 9, 1 / 36, 0], [0, -25 / 216, -20 / 27, 0, 20 / 27, 25 / 216, 0])]
    for e, (lr, rr) in enumerate(edge):
        left[e], right[e] = lr, rr
        left[n - 1 - e], right[n - 1 - e] = lr[::-1], [-v for v in rr[::-1]]
    off = range(-3, 4)
    return _band(left, off, n), _band(right, off, n) / h


def _second_derivative(y):
    """Left and right sides of the compact d2/dy2 on the mesh (cfdiff.f:196-501):
    weights that are exact for the powers of the distance, in local units."""
    n = len(y)
    left, right = np.zeros((n, n)), np.zeros((n, n))
    for j in range(n):
        near = [m for m in (-2, -1, 0, 1, 2) if 0 <= j + m < n]
        lo, ro = [m for m in near if m], near
        u = max(abs(y[j + m] - y[j]) for m in near)
        N = len(lo) + len(ro)
        A, b = np.zeros((N, N)), np.zeros(N)
        for k in range(N):
            for q, m in enumerate(lo):
                A[k, q] = k * (k - 1) * ((y[j + m] - y[j]) / u) ** (k - 2) if k > 1 else 0.0
            for q, m in enumerate(ro):
                A[k, len(lo) + q] = -((y[j + m] - y[j]) / u) ** k if k else -1.0
        b[2] = -2.0
        w = np.linalg.solve(A, b)
        w += np.linalg.solve(A, b - A @ w)
        left[j, j] = 1.0
        for q, m in enumerate(lo):
            left[j, j + m] = w[q]
        for q, m in enumerate(ro):
            right[j, j + m] = w[len(lo) + q] / u**2
    return left, right


class _Plain64:
    def __init__(self, p, y, st, z):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.y, self.dev = p, np.asarray(y), dev
        n = p.my
        c = lambda a: torch.as_tensor(np.ascontiguousarray(np.moveaxis(a, 2, 0))).to(dev)  # noqa: E731
        self.vor, self.phi, self.psi, self.T = (c(st[k]) for k in FIELDS)
        self.Z = c(z) if z is not None else None
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).to(dev)  # noqa: E731
        self.u00, self.v00, self.w00 = (t(st[k]) for k in ("u00", "v00", "w00"))
        self.Twall = (float(st["scal"][0, 0, 0].real), float(st["scal"][0, 0, -1].real))
        self.Zwall = (float(z[0, 0, 0].real), float(z[0, 0, -1].real)) if z is not None else None
        l1, self.r1n = _first_derivative(n)
        l2, r2 = _second_derivative(self.y)
        self.l1n = l1
        fmap = 1.0 / np.linalg.solve(l1, self.r1n @ self.y)
        self.fmapn = fmap
        self.D1 = (t(fmap[:, None] * np.linalg.inv(l1)), t(self.r1n))
        self.D2 = (t(np.linalg.inv(l2)), t(r2))
        self.l2, self.l2n, self.r2n = t(l2), l2, r2
        d = np.diff(self.y)
        self.hyn = 0.5 * (np.append(d, 0.0) + np.append(0.0, d))
        self.hy = t(self.hyn)
        nz1 = (p.mz - 1) // 2
        self.nz1 = nz1
        kz = np.arange(p.mz)
        self.kx = t(p.alp * np.arange(p.nplanes))[:, None]
        self.kz = t(p.bet * np.where(kz <= nz1, kz, kz - p.mz))[None, :]
        self.k2 = self.kx**2 + self.kz**2
        self.inv_k2 = torch.where(self.k2 > 0, 1.0 / self.k2.clamp_min(1e-300), torch.zeros_like(self.k2))
        self._factor(l2, r2)
        self.Rom = self.Rphi = torch.zeros_like(self.vor)
        self.rhsT = self.rhsZ = 0.0
        self.r00 = [torch.zeros_like(self.u00), torch.zeros_like(self.u00)]
        self.dt, self.time, self.diag = p.dt, float(st.get("time", 0.0)), {}
        g, xi = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)
        p0, p1 = 5 / 66, -1.0
        b3 = (p1 * (g[0] * g[2] + g[1] * g[2] + xi[1] * g[2] + g[0] * xi[2]) - g[0] * g[1] * g[2]
              - g[0] * g[1] * xi[2]) / (p1 - g[0] * g[1])
        be = (g[0] - p0, p1, b3)
        self.rk = list(zip(g, xi, (p0, g[1] + xi[1] - p1, g[2] + xi[2] - b3), be))

    # y operators: a pair (A, B) applied as A (B u), all modes at once
    def _y(self, D, f):
        x = torch.view_as_real(f.contiguous()).reshape(f.shape[0], -1) if f.is_complex() else f.reshape(f.shape[0], -1)
        r = D[0] @ (D[1] @ x)
        return torch.view_as_complex(r.reshape(*f.shape, 2)) if f.is_complex() else r.reshape(f.shape)

    def d1(self, f):
        return self._y(self.D1, f)

    def d2(self, f):
        return self._y(self.D2, f)

    def _factor(self, l2, r2):
        """LU of d2 - k2 with identity wall rows, for all modes row by row."""
        n, k2 = self.p.my, self.k2
        row = []
        for j in range(n):
            w = []
            for c in range(j - 2, j + 3):
                if 0 < j < n - 1 and 0 <= c < n:
                    w.append(r2[j, c] - k2 * l2[j, c])
                else:
                    w.append(torch.full_like(k2, 1.0 if c == j else 0.0))
            row.append(w)
        self.low, self.up = [], []
        for j in range(n):
            a = row[j]
            m2 = m1 = None
            if j >= 2:
                u = self.up[j - 2]
                m2 = a[0] * u[0]
                a[1], a[2] = a[1] - m2 * u[1], a[2] - m2 * u[2]
            if j >= 1:
                u = self.up[j - 1]
                m1 = a[1] * u[0]
                a[2], a[3] = a[2] - m1 * u[1], a[3] - m1 * u[2]
            self.low.append((m1, m2))
            self.up.append((1.0 / a[2], a[3], a[4]))
        e = []
        for j in (0, n - 1):
            b = torch.zeros((n,) + tuple(k2.shape), dtype=torch.float64, device=self.dev)
            b[j] = 1.0
            e.append(self._solve(b))
        self.hom = e
        wall = [self.d1(v)[[0, -1]] for v in e]
        det = wall[0][0] * wall[1][1] - wall[1][0] * wall[0][1]
        self.wall = [v / det for v in (wall[1][1], -wall[1][0], -wall[0][1], wall[0][0])]

    def _solve(self, b):
        n = self.p.my
        x = list(b.unbind(0))
        for j in range(1, n):
            m1, m2 = self.low[j]
            x[j] = x[j] - m1 * x[j - 1]
            if j >= 2:
                x[j] = x[j] - m2 * x[j - 2]
        for j in reversed(range(n)):
            p, u1, u2 = self.up[j]
            if j + 1 < n:
                x[j] = x[j] - u1 * x[j + 1]
            if j + 2 < n:
                x[j] = x[j] - u2 * x[j + 2]
            x[j] = x[j] * p
        return torch.stack(x)

    def poisson(self, f, neumann=False):
        b = self._y((self.l2, torch.eye(self.p.my, dtype=torch.float64, device=self.dev)), f)
        b[0] = 0
        b[-1] = 0
        x = self._solve(b)
        if neumann:
            w = self.d1(x)[[0, -1]]
            x = x - (self.wall[0] * w[0] + self.wall[1] * w[1]) * self.hom[0] \
                - (self.wall[2] * w[0] + self.wall[3] * w[1]) * self.hom[1]
        return x * (self.k2 > 0)

    # transforms
    def phys(self, f):
        p, nz1 = self.p, self.nz1
        a = torch.zeros(p.my, p.nplanes, p.mgalz, dtype=torch.complex128, device=self.dev)
        a[..., :nz1 + 1] = f[..., :nz1 + 1]
        if nz1:
            a[..., p.mgalz - nz1:] = f[..., nz1 + 1:]
        a = torch.fft.ifft(a, dim=-1, norm="forward")
        a[:, 0] = a[:, 0].real.to(torch.complex128)
        return torch.fft.irfft(a, n=p.mgalx, dim=1, norm="forward")

    def spec(self, f):
        p, nz1 = self.p, self.nz1
        a = torch.fft.fft(torch.fft.rfft(f, dim=1, norm="forward")[:, :p.nplanes], dim=-1, norm="forward")
        return torch.cat([a[..., :nz1 + 1], a[..., p.mgalz - nz1:]], -1) if nz1 else a[..., :1].contiguous()

    def step(self, cfl_step):
        cfl_step = cfl_step and self.p.dt_mode == 0
        self.diag.update(time=self.time, Deltat=self.dt)
        for r in range(3):
            self.substep(r, cfl_step)
        self.time += self.dt
        if cfl_step:
            self.dt = self.dtr
        self.diag["Deltat_next"] = self.dt

    def substep(self, r, cfl_step):
        p = self.p
        gam, xi, al, be = self.rk[r]
        dtx, dtg, dtb = self.dt * xi, self.dt * gam, self.dt * be
        ikx, ikz, k2 = 1j * self.kx, 1j * self.kz, self.k2
        ire, ipe, ipz = 1.0 / p.Re, 1.0 / (p.Re * PR), 1.0 / (p.Re * PR)
        vor, phi, T = self.vor.clone(), self.phi.clone(), self.T.clone()
        vor[0], vor[-1] = vor[1].clone(), vor[-2].clone()
        for f, wall in ((phi, None), (T, self.Twall), (self.Z, self.Zwall)):
            if f is not None:
                f[0] = 0
                f[-1] = 0
                if wall:
                    f[0, 0, 0], f[-1, 0, 0] = wall
        my_ = self.poisson(phi)
        dmy = self.d1(my_)
        ru = ikx * (self.psi + dmy * self.inv_k2) - ikz * self.inv_k2 * vor
        rw = ikz * (self.psi + dmy * self.inv_k2) + ikx * self.inv_k2 * vor
        rv = my_ + self.d1(self.psi)
        for f, m in ((ru, self.u00), (rv, self.v00), (rw, self.w00)):
            f[:, 0, 0] = m.to(torch.complex128)
        del my_, dmy
        self.u00[1:-1] += dtx * self.r00[0][1:-1]
        self.w00[1:-1] += dtx * self.r00[1][1:-1]
        vor, phi = vor + dtx * self.Rom, phi + dtx * self.Rphi
        ph = self.phys
        pu, pv, pw, pT = ph(ru), ph(rv), ph(rw), ph(T)
        tx, ty, tz, lapT = ph(ikx * T), ph(self.d1(T)), ph(ikz * T), ph(self.d2(T) - k2 * T)
        u, v, w = pu * pT, pv * pT, pw * pT
        grad2 = pT * lapT
        tsg = 1.0
        if p.visc:
            tsg = pT**p.sigma
            grad2 = tsg * (grad2 + p.sigma * (tx * tx + ty * ty + tz * tz))
        rhs = -u * tx - v * ty - w * tz + grad2 * ipe
        d8 = dtx * self.rhsT + dtg * rhs
        dZ = None
        if self.Z is not None:
            Z = self.Z
            zx, zy, zz = ph(ikx * Z), ph(self.d1(Z)), ph(ikz * Z)
            lz = pT * ph(self.d2(Z) - k2 * Z)
            if p.visc:
                lz = tsg * (lz + p.sigma * (tx * zx + ty * zy + tz * zz))
            rz = -u * zx - v * zy - w * zz + lz * ipz
            dZ = self.spec(dtx * self.rhsZ + dtg * rz)
            self.rhsZ = rz
            del zx, zy, zz, lz, rz
        s = self.spec
        U, V, W = s(u), s(v), s(w)

        def stress(a, b, g, sym):
            """rho u_i u_j less the variable part of the stress."""
            if not p.visc:
                return s(a * b)
            return s(a * b - ire * (tsg - 1.0) * (pT * ph(g) + sym))
        uu = stress(pu, u, 2 * ikx * ru, 2 * pu * tx)
        vv = stress(pv, v, 2 * self.d1(rv) if p.visc else None, 2 * pv * ty)
        ww = stress(pw, w, 2 * ikz * rw, 2 * pw * tz)
        uv = stress(pu, v, self.d1(ru) + ikx * rv if p.visc else None, pu * ty + pv * tx)
        uw = stress(pu, w, ikz * ru + ikx * rw, pu * tz + pw * tx)
        vw = stress(pv, w, ikz * rv + self.d1(rw) if p.visc else None, pv * tz + pw * ty)
        drho = s((d8 / (pT * (pT + d8))) / dtb - (al / be) * rhs / (pT * pT))
        self.T = T + s(d8)
        if dZ is not None:
            self.Z = self.Z + dZ
        self.rhsT = rhs
        u00 = U[:, 0, 0].real.clone()
        w00 = W[:, 0, 0].real.clone()
        if r == 0:
            a = torch.cat([u00[1:], u00[-1:]])
            b = torch.cat([u00[:1], u00[:-1]])
            sm = float((0.5 * self.hy * (a * a + b * b)).sum())
            self.diag["dm"] = 0.25 * (self.y[-1] - self.y[0]) - sm / float(u00[-1] - u00[0]) ** 2
            self.diag["masst"] = float(((1.0 / pT).mean(dim=(1, 2)) * self.hy).sum())
            if cfl_step:
                hx, hz = p.alp * (p.mgalx - 1) / math.pi, p.bet * (p.mgalz - 1) / math.pi
                big = lambda q: q.abs().amax(dim=(1, 2))  # noqa: E731
                Tm = pT.amax(dim=(1, 2))
                D = ipe * (Tm ** (1.0 + p.sigma) if p.visc else Tm)
                ct = (2 * D * ((hx / 2) ** 2 + (hz / 2) ** 2 + 1.0 / self.hy**2)).max()
                reig = big(u).max() * hx / 2 + (big(v) / self.hy).max() + big(w).max() * hz / 2 + ct
                self.dtr = float(np.float32(float(np.float32(p.cfl)) / float(reig)))
        del pu, pv, pw, pT, tx, ty, tz, lapT, u, v, w, grad2, tsg, rhs, d8
        Ny = -ikx * uv - self.d1(vv) - ikz * vw
        duv, dvw = self.d1(uv), self.d1(vw)
        Nx = -ikx * uu - duv - ikz * uw
        Nz = -ikx * uw - dvw - ikz * ww
        self.r00 = [-duv[:, 0, 0].real + ire * self.d2(u00[:, None])[:, 0],
                    -dvw[:, 0, 0].real + ire * self.d2(w00[:, None])[:, 0]]
        if r == 2:
            dw = 1.0 / float(self.d1(u00[:, None]).abs().max())
            self.diag.update(dw=dw, Redw=dw / ire, H00u=0.25 * float((self.r00[0] * self.hy).sum()),
                             H00w=0.25 * float((self.r00[1] * self.hy).sum()))
        ox = self.d1(W) - ikz * V
        oz = ikx * V - self.d1(U)
        oy = ikz * U - ikx * W
        cy = ikz * ox - ikx * oz
        self.Rom = ikz * Nx - ikx * Nz + ire * (self.d2(oy) - k2 * oy)
        self.Rphi = -k2 * Ny - self.d1(ikx * Nx + ikz * Nz) - ire * (self.d2(cy) - k2 * cy)
        self.vor, self.phi = vor + dtg * self.Rom, phi + dtg * self.Rphi
        self.psi = self.poisson(drho, neumann=True)
        self.u00[1:-1] += dtg * self.r00[0][1:-1]
        self.w00[1:-1] += dtg * self.r00[1][1:-1]
        self.diag.update(massu=float((self.u00 * self.hy).sum()), massv=float((self.v00 * self.hy).sum()),
                         massw=float((self.w00 * self.hy).sum()))
        # rho v00: the integral of d(rho)/dt (laps.f:484-575) and the wall correction
        q = self.l1n @ (drho[:, 0, 0].real.cpu().numpy() / self.fmapn)
        f = np.append(np.linalg.solve(self.r1n[:-1, :-1], q[:-1]), 0.0)
        f -= f[0]
        trapz = -f[-1]
        self.diag["trapz"] = trapz
        self.v00 = torch.as_tensor(f + trapz / (1.0 + math.sqrt(self.Twall[0] / self.Twall[1]))).to(self.dev)

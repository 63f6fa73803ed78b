"""Cases of the work a user has this library do, with inputs, one pass and its 64-bit result.

  step      restart from a state kept on the device and advance it `steps` time steps
            (wf_step: RK stages, pressure solve, projection), the main loop of a run
  host      the same from host buffers: upload, one step, download (a program that
            keeps its fields on the host, as the reference's does)
  ensemble  independent scenarios of uneven grids advanced together
  phi, rk, pressure
            the reference's operators on the caller's device buffers (wf_phi_device,
            wf_rk_device, wf_pressure_device), which the drop-in's Phi, RK4 and
            solve_pressure call

Grids are those of the benchmark (512 x 512 x 128 eight hills, 256 x 256 x 128,
128 x 128 x 64 flat, ensemble members of 96 to 256 points) and of the tests
(33 x 33 x 16), and ragged ones between.  Physics: "inert" is the benchmark's
setting (constant density, no convective exchange or drag), "full" has drag,
convective exchange and the Sutherland laws, "vardens" the reference's default
variable density (fixed point to 1e-10, at most 50 solves) and "closure" the
learned subgrid closure in place of C_s^2.
"""
import ctypes as C
import math
import os
import random
import tempfile

import numpy as np
import torch

DX, DT = 1.5625, 0.003
T_INF, T_PC, T_ACT, A_RR, H_C, C_P = 300.0, 523.0, 18040.8533, 1e9, 21e6, 1007.0
MU, K_T, RHO, GRAV, DELTA, PR, Y_F, Y_H = 1.802e-5, 0.02476, 1.1, -9.807, 0.1, 0.7329, 100.0, 0.8
C_S, C_D, HCONV, T_MAX, TOL, MAXIT = 0.173, 0.15, 1.42, 2500.0, 1e-10, 50
SIGMA_SB = 5.670374419e-8
FIELDS = ("u", "v", "w", "T", "Y")


def _case(name, kind, Nx, Ny, Nz, prec, physics="inert", method="RK4", hills=0, stretch=0.0, steps=1, members=1):
    return {"name": name, "kind": kind, "Nx": Nx, "Ny": Ny, "Nz": Nz, "prec": prec, "physics": physics,
            "method": method, "hills": hills, "stretch": stretch, "steps": steps, "members": members}


def listed():
    return [
        # the benchmark's headline workload: FP32 stencil on the full grid
        _case("hills8_512_fp32", "step", 512, 512, 128, "fp32", hills=8),
        # the plain FP64 path on the single-hill workload's grid
        _case("hill_256_fp64", "step", 256, 256, 128, "fp64", hills=1),
        # the flat workload, several steps between two looks at the state
        _case("flat_128_fp32", "step", 128, 128, 64, "fp32", steps=5),
        # the smallest grid in use (debugging, coupling tests): latency and launches
        _case("flat_33_fp64", "step", 33, 33, 16, "fp64", steps=10),
        # a user's own grid: odd sizes, stretched z, RK2, all source terms on
        _case("ragged_201x150x45_fp32", "step", 201, 150, 45, "fp32", "full", "RK2", hills=3, stretch=1.5, steps=2),
        # the reference's default variable density
        _case("vardens_160x128x48_fp32", "step", 160, 128, 48, "fp32", "vardens", hills=2),
        # learned subgrid closure
        _case("closure_128x128x32_fp32", "step", 128, 128, 32, "fp32", "closure", steps=2),
        # scenario ensemble of uneven grids
        _case("ensemble_10_fp32", "ensemble", 96, 256, 64, "fp32", hills=2, members=10),
        # fields kept on the host: upload, step, download
        _case("host_256x256x64_fp32", "host", 256, 256, 64, "fp32", hills=1),
        # the drop-in's operators on device buffers
        _case("phi_191x96x50_fp64", "phi", 191, 96, 50, "fp64", "full", hills=2),
        _case("pressure_257x200x64_fp64", "pressure", 257, 200, 64, "fp64"),
        _case("rk_300x260x64_fp32", "rk", 300, 260, 64, "fp32", hills=4),
    ]


def draw(rng):
    """A case of the same ranges: 17 to 512 points in x and y, 12 to 160 in z, at most 9 million cells (an
    ensemble: 5 million in all), either precision, any method, terrain, physics and kind."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["step", "step", "step", "step", "phi", "rk", "pressure", "ensemble", "host"])
    prec = rng.choice(["fp32", "fp32", "fp64"])
    physics = rng.choice(["inert", "inert", "inert", "full", "vardens", "closure"])
    members = 1
    if kind == "ensemble":
        members = rng.randint(3, 8)
        Nx, Ny, Nz, most = size(48, 96), size(100, 200), rng.choice([32, 48, 64, 57]), 5e6 / members
    else:
        Nx, Ny, Nz, most = size(17, 512), size(17, 512), size(12, 160), 9e6
    while Nx * Ny * Nz > most:
        Nx, Ny, Nz = max(17, int(Nx * 0.93)), max(17, int(Ny * 0.93)), max(12, int(Nz * 0.97))
    if physics == "vardens" and (kind not in ("step", "pressure") or Nx * Ny * Nz > 2e6):
        physics = "inert"
    if physics == "closure" and kind != "step":
        physics = "inert"
    c = _case("", kind, Nx, Ny, Nz, prec, physics, rng.choice(["RK4", "RK4", "RK4", "RK2", "Euler"]),
              rng.randint(0, 6), rng.choice([0.0, 0.0, 1.0, 2.0]),
              rng.choice([1, 2, 5]) if kind == "step" and Nx * Ny * Nz < 1e6 else 1, members)
    del c["name"]
    return c


def _sizes(case):
    """Grid sizes of the members: one grid, or an ensemble's between its smallest and largest size."""
    if case["kind"] != "ensemble":
        return [(case["Nx"], case["Ny"], case["Nz"])]
    r = random.Random(case["members"] * 1000 + case["Nx"])
    lo, hi = case["Nx"], case["Ny"]
    some = sorted({lo, hi, (2 * lo + hi) // 3, (lo + 2 * hi) // 3, (lo + hi) // 2})
    return [(r.choice(some), r.choice(some), case["Nz"]) for _ in range(case["members"])]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


# ---- inputs ---------------------------------------------------------------------
def _hills(case, size):
    """Gaussian hills (centre x, centre y, height, width) of a grid, the same for every seed (the terrain sets the
    stored fuel layer's size); in metres, 2 to 12% of the box's height."""
    r = random.Random(size[0] * 7919 + size[1] * 104729 + size[2])
    Lx, Ly, H = (size[0] - 1) * DX, (size[1] - 1) * DX, _height(size[2])
    return [(r.uniform(0, Lx), r.uniform(0, Ly), H * r.uniform(0.02, 0.12), r.uniform(0.05, 0.12) * min(Lx, Ly))
            for _ in range(case["hills"])]


def _height(Nz):
    return 0.47 * (Nz - 1)


def _z(case, Nz):
    H = _height(Nz)
    k = np.arange(Nz)
    if case["stretch"]:
        dz = H / (Nz - 1)
        return H * (np.exp(case["stretch"] * k * dz / H) - 1) / (math.exp(case["stretch"]) - 1)
    return k * (H / (Nz - 1))


def _terrain(case, size, dev):
    """Terrain height, cut nodes and fuel tops of the columns, [Nx, Ny]."""
    Nx, Ny, Nz = size
    Lx, Ly = (Nx - 1) * DX, (Ny - 1) * DX
    x = (torch.arange(Nx, device=dev, dtype=torch.float64) * (Lx / (Nx - 1)))[:, None]
    y = (torch.arange(Ny, device=dev, dtype=torch.float64) * (Ly / (Ny - 1)))[None, :]
    h = torch.zeros(Nx, Ny, device=dev, dtype=torch.float64)
    for cx, cy, hh, wd in _hills(case, size):
        dx = torch.remainder(x - cx + Lx / 2, Lx) - Lx / 2
        dy = torch.remainder(y - cy + Ly / 2, Ly) - Ly / 2
        h = h + hh * torch.exp(-(dx * dx + dy * dy) / (2 * wd * wd))
    z = torch.tensor(_z(case, Nz), device=dev)
    dz = torch.cat([z[1:] - z[:-1], (z[-1] - z[-2])[None]])
    k = torch.arange(Nz, device=dev)
    at = (h[..., None] - dz <= z) & (z <= h[..., None])
    cut = torch.where(at, k, 0).amax(-1)
    nzy = torch.where(z <= h[..., None] + Y_H, k + 1, 0).amax(-1)
    return h, cut, nzy


def _fields(case, size, seed, dev):
    """Seeded state: log wind above the terrain with gusts, three burning spots, uneven fuel.  Values are
    single-precision numbers, so both precisions start from the same state.  [u, v, w, T, Y] and p."""
    Nx, Ny, Nz = size
    h, cut, nzy = _terrain(case, size, dev)
    g = torch.Generator(device=dev).manual_seed(seed + 1)
    r = random.Random(seed * 31 + 5)
    z = torch.tensor(_z(case, Nz), device=dev)
    hgt = z - h[..., None]
    speed = r.uniform(3, 8) * torch.log(hgt.clamp(min=0.05) / 0.05) / math.log(2.0 / 0.05)
    th = r.uniform(0, 2 * math.pi)

    def gust(a):   # white noise smoothed over a few cells
        n = torch.randn(Nx - 1, Ny - 1, Nz, generator=g, device=dev, dtype=torch.float32)
        n = (n + n.roll(1, 0) + n.roll(-1, 0)) / 3
        n = (n + n.roll(1, 1) + n.roll(-1, 1)) / 3
        return a * torch.cat([torch.cat([n, n[:, :1]], 1), torch.cat([n[:1], n[:1, :1]], 1)], 0).double()

    u, v, w = speed * math.cos(th) + gust(0.3), speed * math.sin(th) + gust(0.3), gust(0.15)
    Lx, Ly = (Nx - 1) * DX, (Ny - 1) * DX
    x = (torch.arange(Nx, device=dev, dtype=torch.float64) * DX)[:, None]
    y = (torch.arange(Ny, device=dev, dtype=torch.float64) * DX)[None, :]
    heat = torch.zeros(Nx, Ny, device=dev, dtype=torch.float64)
    for _ in range(3):
        cx, cy = r.uniform(0, Lx), r.uniform(0, Ly)
        dx = torch.remainder(x - cx + Lx / 2, Lx) - Lx / 2
        dy = torch.remainder(y - cy + Ly / 2, Ly) - Ly / 2
        heat = torch.maximum(heat, 500.0 * torch.exp(-(dx * dx + dy * dy) / (2 * 3.0 ** 2)))
    T = T_INF + torch.where(hgt < 1.0, heat[..., None], 0.0) + gust(0.5).abs()
    k = torch.arange(Nz, device=dev)
    dead = k < cut[..., None]
    u, v, w = (torch.where(dead, 0.0, f) for f in (u, v, w))
    T = torch.where(dead, T_INF, T)
    Yc = 0.5 + 0.5 * torch.rand(Nx, Ny, generator=g, device=dev, dtype=torch.float32).double()
    NzY = int(nzy.max())
    Y = torch.where((k < nzy[..., None]) & ~dead, Yc[..., None], 0.0)[:, :, :NzY]
    out = []
    for f in (u, v, w, T, Y):
        f = f.float().double()
        f[-1], f[:, -1] = f[0], f[:, 0]
        out.append(f)
    return out, torch.zeros(Nx, Ny, Nz, device=dev, dtype=torch.float64)


def _packed(fields):
    return torch.cat([f.reshape(-1) for f in fields])


def _params(case, size):
    from wildfires_b200 import read_parameters
    Nx, Ny, Nz = size
    full = case["physics"] == "full"
    d = dict(Nx=Nx, Ny=Ny, Nz=Nz, Nt=1000, NT=1000, x_min=0.0, x_max=(Nx - 1) * DX, y_min=0.0, y_max=(Ny - 1) * DX,
             z_min=0.0, z_max=_height(Nz), t_min=0.0, t_max=1000 * DT, method=case["method"], rho_inf=RHO, C_s=C_S,
             T_inf=T_INF, T_dead_nodes=T_INF, Y_f=Y_F, Y_h=Y_H, p_top=0.0, alpha_s=0.002 if full else 0.0,
             sigma_s=5500.0 if full else 0.0, sutherland_viscosity=int(full), sutherland_conductivity=int(full),
             variable_density=int(case["physics"] == "vardens"), pressure_solver_iter=MAXIT, pressure_solver_tol=TOL,
             t_source_start=0.0, t_source_end=0.0, topo_shape="flat", Y0_x_start=0.0, Y0_x_end=(Nx - 1) * DX,
             Y0_y_start=0.0, Y0_y_end=(Ny - 1) * DX, temperature_convection=1, velocity_correction_fd=0,
             time_step_log=1000000, z_domain=1 if case["stretch"] else 0, k_nu_grid=case["stretch"])
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "parameters.txt")
        with open(path, "w") as f:
            f.write("".join("%s = %s\n" % (k, v if isinstance(v, str) else repr(v)) for k, v in d.items()))
        P = read_parameters(path)
    hills = _hills(case, size)
    if hills:
        P.set_topography_hills(hills)
    return P


def _weights(seed):
    from wildfires_b200 import closure
    return closure.init_params(seed)


class _DeviceArray:
    """A solver's device buffer; a tensor over it keeps the solver (its owner) alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _view(owner, solver, keep):
    """Tensors over a solver's current device state and pressure, kept per buffer."""
    y, p = solver.device_state()
    if y not in keep:
        kind = "<f4" if solver.precision == "fp32" else "<f8"
        keep[y] = (torch.as_tensor(_DeviceArray(owner, y, solver.S, kind), device="cuda"),
                   torch.as_tensor(_DeviceArray(owner, p, solver.N, "<f8"), device="cuda"))
    return keep[y]


def _split(y, size):
    """The packed state's fields."""
    Nx, Ny, Nz = size
    N = Nx * Ny * Nz
    out = {f: y[q * N:(q + 1) * N].reshape(Nx, Ny, Nz) for q, f in enumerate("uvwT")}
    out["Y"] = y[4 * N:].reshape(Nx, Ny, -1)
    return out


# ---- a case's state and one pass ---------------------------------------------------
def prepare(case, seed):
    from wildfires_b200 import Ensemble, Solver, _abi
    sizes = _sizes(case)
    Ps = [_params(case, sz) for sz in sizes]
    ins = [_fields(case, sz, seed + 17 * m, "cuda") for m, sz in enumerate(sizes)]
    s = {"case": case, "sizes": sizes, "lib": _abi.lib(), "check": _abi.check}
    if case["kind"] == "ensemble":
        s["solver"] = Ensemble(Ps, case["prec"])
        s["members"] = s["solver"].members
    else:
        s["solver"] = Solver(Ps[0], case["prec"])
        s["members"] = [s["solver"]]
        if case["physics"] == "closure":
            th = _weights(seed)
            _abi.check(s["lib"].wf_set_closure(s["solver"]._h, 1, th.ctypes.data_as(C.POINTER(C.c_float))), "wf_set_closure")
    s["stream"] = torch.cuda.ExternalStream(s["solver"].stream())
    s["views"] = [{} for _ in sizes]
    ys = [_packed(f) for f, _ in ins]
    if case["kind"] in ("step", "ensemble"):
        for m, y in zip(s["members"], ys):
            m.upload(y.cpu().numpy(), np.zeros(m.N))
        s["y0"] = [y.float() if case["prec"] == "fp32" else y for y in ys]
        s["p0"] = [p.reshape(-1) for _, p in ins]
    elif case["kind"] == "host":
        s["y"], s["p"] = (torch.empty(n, dtype=torch.float64, pin_memory=True) for n in (s["solver"].S, s["solver"].N))
        s["y1"], s["p1"] = (torch.empty(n, dtype=torch.float64, pin_memory=True) for n in (s["solver"].S, s["solver"].N))
        s["y"].copy_(ys[0])
        s["p"].zero_()
    else:
        s["y"], s["out"], s["p"] = ys[0], torch.zeros_like(ys[0]), ins[0][1].reshape(-1)
        s["p1"] = torch.zeros_like(s["p"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind, solver, L = s["case"]["kind"], s["solver"], s["lib"]
    vp = C.c_void_p
    if kind in ("step", "ensemble"):
        with torch.cuda.stream(s["stream"]):
            for m, keep, y0, p0 in zip(s["members"], s["views"], s["y0"], s["p0"]):
                y, p = _view(solver, m, keep)
                y.copy_(y0)
                p.copy_(p0)
        solver.step(s["case"]["steps"])
        out = []
        for m, keep, size in zip(s["members"], s["views"], s["sizes"]):
            y, p = _view(solver, m, keep)
            out.append(dict(_split(y, size), p=p))
        return out
    if kind == "host":
        dp = C.POINTER(C.c_double)
        h = [C.cast(s[k].data_ptr(), dp) for k in ("y", "p", "y1", "p1")]
        s["check"](L.wf_upload_state_async(solver._h, h[0], h[1]), "wf_upload_state_async")
        solver.step(1)
        s["check"](L.wf_download_state(solver._h, h[2], h[3]), "wf_download_state")
        return [dict(_split(s["y1"].numpy(), s["sizes"][0]), p=s["p1"].numpy())]
    y, out = vp(s["y"].data_ptr()), vp(s["out"].data_ptr())
    if kind == "phi":
        s["check"](L.wf_phi_device(solver._h, y, out), "wf_phi_device")
        return [_split(s["out"], s["sizes"][0])]
    if kind == "rk":
        s["check"](L.wf_rk_device(solver._h, y, out), "wf_rk_device")
        return [_split(s["out"], s["sizes"][0])]
    with torch.cuda.stream(s["stream"]):
        s["p1"].copy_(s["p"])
    s["check"](L.wf_pressure_device(solver._h, y, y, vp(s["p1"].data_ptr())), "wf_pressure_device")
    return [{"p": s["p1"]}]


def work(case):
    """Bytes and operations of a pass.  A stage reads its input and its RK operands once and writes its outputs
    once (their sum over a step: 17 state passes for RK4, 7 for RK2, 2 for Euler); a pressure solve reads u, v, w
    and writes p with the spectrum passing through memory five times each way; the projection reads p and the state
    and writes u, v, w.  Operations: 300 per cell and stage, 5 n log2 n per transform.  Host copies are not counted."""
    e = 4 if case["prec"] == "fp32" else 8
    stages, passes = {"RK4": (4, 17), "RK2": (2, 7), "Euler": (1, 2)}[case["method"]]
    total = {"bytes": 0.0, "flops": 0.0}
    for Nx, Ny, Nz in _sizes(case):
        N = Nx * Ny * Nz
        solves = 20 if case["physics"] == "vardens" else 1
        b_solve, f_solve = solves * (3 * e + 9 * 8 + 8) * N, solves * N * (5 * math.log2(Nx * Ny) + 20)
        b_rk, f_rk = 4 * passes * e * N, 300 * stages * N
        if case["physics"] == "closure":
            f_rk += stages * N * 2 * (12 * 64 + 64 * 64 + 64)
        if case["kind"] == "phi":
            b, f = 8 * 8 * N, 300 * N
        elif case["kind"] == "rk":
            b, f = b_rk, f_rk
        elif case["kind"] == "pressure":
            b, f = b_solve, f_solve
        else:
            b, f = b_rk + b_solve + (8 + 7 * e) * N, f_rk + f_solve
            b, f = b * case["steps"], f * case["steps"]
        total["bytes"] += b
        total["flops"] += f
    return total


# ---- the model in 64 bits ------------------------------------------------------------
class _Exact:
    """The model's operators in plain torch, on the unique cells of the periodic grid (Nx-1 x Ny-1 x Nz)."""

    def __init__(self, case, size, seed, dev):
        self.case, (self.Nx, self.Ny, self.Nz) = case, size
        self.full, self.vardens = case["physics"] == "full", case["physics"] == "vardens"
        h, cut, nzy = (t[:-1, :-1] for t in _terrain(case, size, dev))
        self.NzY = int(nzy.max())
        self.topo, self.cut, self.nzy = h[..., None], cut[..., None], nzy[..., None]
        self.k = torch.arange(self.Nz, device=dev)
        self.z = z = torch.tensor(_z(case, self.Nz), device=dev)
        self.d = d = z[1:] - z[:-1]
        self.dz = torch.cat([d, d[-1:]])
        self.fuel = self.k < self.nzy
        self.dead, self.live = self.k < self.cut, (self.k > self.cut) & (self.k < self.Nz - 1)
        self.theta = None
        if case["physics"] == "closure":
            th = torch.tensor(_weights(seed), device=dev).double()
            o = 0
            self.theta = []
            for shape in ((64, 12), (64,), (64, 64), (64,), (64,), (1,), (12,)):
                n = math.prod(shape)
                self.theta.append(th[o:o + n].reshape(shape))
                o += n

    # derivatives
    def x(self, f):
        return (f.roll(-1, 0) - f.roll(1, 0)) / (2 * DX)

    def y(self, f):
        return (f.roll(-1, 1) - f.roll(1, 1)) / (2 * DX)

    def lap(self, f):
        return ((f.roll(-1, 0) - 2 * f + f.roll(1, 0)) + (f.roll(-1, 1) - 2 * f + f.roll(1, 1))) / (DX * DX) + self.zz(f)

    def _fwd(self, f):   # one-sided at k, from k, k+1, k+2 (k <= Nz-3)
        a, b = self.d[:-1], self.d[1:]
        return -(2 * a + b) / (a * (a + b)) * f[..., :-2] + (a + b) / (a * b) * f[..., 1:-1] - a / (b * (a + b)) * f[..., 2:]

    def _bwd(self, f):   # from k-2, k-1, k (k >= 2)
        a2, a1 = self.d[:-1], self.d[1:]
        return a1 / (a2 * (a2 + a1)) * f[..., :-2] - (a2 + a1) / (a2 * a1) * f[..., 1:-1] + (a2 + 2 * a1) / (a1 * (a2 + a1)) * f[..., 2:]

    def zd(self, f):     # central, one-sided at the walls
        c = (f[..., 2:] - f[..., :-2]) / (self.d[:-1] + self.d[1:])
        return torch.cat([self._fwd(f)[..., :1], c, self._bwd(f)[..., -1:]], -1)

    def zz(self, f):
        a1, a = self.d[:-1], self.d[1:]
        c = 2 / (a1 * (a1 + a)) * f[..., :-2] - 2 / (a1 * a) * f[..., 1:-1] + 2 / (a * (a1 + a)) * f[..., 2:]
        a, b, e = self.d[0], self.d[1], self.d[2]
        lo = ((6 * a + 4 * b + 2 * e) / (a * (a + b) * (a + b + e)) * f[..., 0] - (4 * a + 4 * b + 2 * e) / (a * b * (b + e)) * f[..., 1]
              + (4 * a + 2 * b + 2 * e) / (b * e * (a + b)) * f[..., 2] - (4 * a + 2 * b) / (e * (b + e) * (a + b + e)) * f[..., 3])
        a1, a2, a3 = self.d[-1], self.d[-2], self.d[-3]
        hi = (-(2 * a2 + 4 * a1) / (a3 * (a3 + a2) * (a3 + a2 + a1)) * f[..., -4] + (2 * a3 + 2 * a2 + 4 * a1) / (a3 * a2 * (a2 + a1)) * f[..., -3]
              - (2 * a3 + 4 * a2 + 4 * a1) / (a2 * a1 * (a3 + a2)) * f[..., -2] + (2 * a3 + 4 * a2 + 6 * a1) / (a1 * (a2 + a1) * (a3 + a2 + a1)) * f[..., -1])
        return torch.cat([lo[..., None], c, hi[..., None]], -1)

    def advect(self, U, f):
        out = torch.zeros_like(f)
        for ax in (0, 1):
            a = (3 * f - 4 * f.roll(1, ax) + f.roll(2, ax)) / (2 * DX)
            b = (-3 * f + 4 * f.roll(-1, ax) - f.roll(-2, ax)) / (2 * DX)
            out += U[ax].clamp(min=0) * a + U[ax].clamp(max=0) * b
        F, B = self._fwd(f), self._bwd(f)
        up = torch.cat([F[..., :2], B], -1)
        down = torch.cat([F, B[..., -2:]], -1)
        return out + U[2].clamp(min=0) * up + U[2].clamp(max=0) * down

    def _arrhenius(self, T):
        return torch.where(T > T_PC, A_RR * torch.exp(-T_ACT / T), 0.0)

    def _pad(self, Y):
        out = torch.zeros(Y.shape[0], Y.shape[1], self.Nz, device=Y.device, dtype=Y.dtype)
        out[..., :self.NzY] = Y
        return torch.where(self.fuel, out, 0.0)

    def _coef(self, u, v, w, T):
        """The learned coefficient in place of C_s^2."""
        W1, b1, W2, b2, W3, b3, sc = self.theta
        s = (DX * DX * self.dz) ** (1.0 / 3.0)
        g = [[self.x(f), self.y(f), self.zd(f)] for f in (u, v, w, T)]
        F = [g[0][0] * s, g[1][1] * s, g[2][2] * s, 0.5 * (g[0][1] + g[1][0]) * s, 0.5 * (g[0][2] + g[2][0]) * s,
             0.5 * (g[1][2] + g[2][1]) * s, (g[2][1] - g[1][2]) * s, (g[0][2] - g[2][0]) * s, (g[1][0] - g[0][1]) * s,
             g[3][0] * s * 0.01, g[3][1] * s * 0.01, g[3][2] * s * 0.01]
        F = torch.stack(F, -1)
        F[:, :, 0] = 0.0
        F[:, :, -1] = 0.0
        gelu = torch.nn.functional.gelu
        a = gelu((F * sc) @ W1.T + b1, approximate="tanh")
        a = gelu(a @ W2.T + b2, approximate="tanh")
        return torch.nn.functional.softplus(a @ W3 + b3)

    def phi(self, u, v, w, T, Y):
        U = (u, v, w)
        Yp = self._pad(Y)
        rho = RHO * T_INF / T
        mu = MU * torch.ones_like(T)
        kT, dk = K_T, 0.0
        if self.full:
            x = T / 273.15
            mu = 1.716e-5 * x ** 1.5 * (273.15 + 110.4) / (T + 110.4)
            kT = 0.0241 * x ** 1.5 * (273.15 + 194) / (T + 194)
            dk = 0.0241 * (1.5 * x ** 0.5 * (273.15 + 194) / (T + 194) - x ** 1.5 * (273.15 + 194) / (T + 194) ** 2)
        Tx, Ty, Tz, lapT = self.x(T), self.y(T), self.zd(T), self.lap(T)
        K = self._arrhenius(T)
        q = H_C / C_P * Yp * K
        cd = 0.0
        if self.full:
            a_s = 0.002 * 5500.0
            cd = 0.5 * C_D * a_s
            zone = self.k <= self.nzy
            Tg = torch.where(zone & ~(Yp > 0), T, T_INF)
            Ts = torch.where(zone & (Yp > 0), T, T_INF)
            hc = HCONV * self.dz * ((Tg - Ts).abs() / self.dz) ** 0.25
            q = q - hc * a_s * (Tg - Ts) / (C_P * T_INF * RHO / Tg)
        src = (dk + 12 * SIGMA_SB * DELTA * T * T * (Tx * Tx + Ty * Ty + Tz * Tz) + (kT + 4 * SIGMA_SB * DELTA * T ** 3) * lapT) / (rho * C_P) + q
        nu = mu / rho
        # subgrid inputs
        g = [[self.x(f), self.y(f), self.zd(f)] for f in U]
        ux, uy, uz, vx, vy, vz, wx, wy, wz = (g[a][b] for a in range(3) for b in range(3))
        S = {(0, 0): (2 * ux - vy - wz) / 3, (1, 1): (2 * vy - ux - wz) / 3, (2, 2): (2 * wz - ux - vy) / 3,
             (0, 1): (uy + vx) / 2, (0, 2): (uz + wx) / 2, (1, 2): (wy + vz) / 2}
        mod_S = torch.sqrt(2 * (ux * ux + vy * vy + wz * wz) + (uz + wx) ** 2 + (vx + uy) ** 2 + (wy + vz) ** 2)
        if self.theta is None:
            ms = rho * (C_S * (DX * DX * self.dz) ** (1.0 / 3.0)) ** 2 * mod_S
        else:
            ms = rho * (DX * DX * self.dz) ** (2.0 / 3.0) * self._coef(u, v, w, T) * mod_S
        divU = nu * src / T
        # Van Driest damping: the neighbour's wall distance and friction, this cell's viscosity
        wall = torch.sqrt((mu[..., 0] * self._fwd(u)[..., 0]) ** 2 + (mu[..., 0] * self._fwd(v)[..., 0]) ** 2)
        ut = torch.sqrt(wall / rho[..., 0])[..., None]
        damp = (self.z - self.topo).clamp(min=0) * ut / 26.0

        def mud(s, ax):
            return ms.roll(-s, ax) * (1 - torch.exp(-damp.roll(-s, ax) * rho / MU)) ** 2

        c = mud(0, 0)
        mx = (mud(1, 0) - mud(-1, 0)) / (2 * DX)
        my = (mud(1, 1) - mud(-1, 1)) / (2 * DX)
        hz = torch.ones_like(self.z)
        hz[1:-1] = self.d[:-1] + self.d[1:]
        mz = (mud(1, 2) - mud(-1, 2)) / hz       # the wall planes are not used
        k = []
        for i in range(3):
            s = [S[min(i, j), max(i, j)] for j in range(3)]
            sgs = -2 * (mx * s[0] + my * s[1] + mz * s[2] + c * (self.x(s[0]) + self.y(s[1]) + self.zd(s[2]))) / rho
            grad = (self.x, self.y, self.zd)[i](divU) / 3
            k.append(nu * self.lap(U[i]) - self.advect(U, U[i]) - sgs + grad)
        if self.full:
            mod_U = torch.sqrt(u * u + v * v + w * w)
            k = [a - cd * Yp * mod_U * b for a, b in zip(k, U)]
        k[2] = k[2] + GRAV * (rho - RHO) / rho
        k.append(src - self.advect(U, T) + (mx * Tx + my * Ty + mz * Tz + c * lapT) / (rho * PR))
        kY = torch.where(self.fuel, -Y_F * K * Yp, 0.0)
        # boundary rules: the cut node, the top, the dead nodes (their k-values are the dead values)
        k, kY = [torch.where(self.live, a, 0.0) for a in k], torch.where(self.k > self.cut, kY, 0.0)
        return self._walls(k, kY, [0.0, 0.0, 0.0, T_INF])

    def _walls(self, f, Y, dead):
        """Boundary rules on fields [u, v, w, T] and fuel Y [.., Nz] with the live values in place."""
        cut = self.cut
        A, B = self.z[cut + 1] - self.z[cut], self.z[cut + 2] - self.z[cut + 1]

        def node(g):
            return ((A + B) ** 2 * g.gather(2, cut + 1) - A * A * g.gather(2, cut + 2)) / (B * (2 * A + B))

        vals = [torch.zeros_like(A), torch.zeros_like(A), torch.zeros_like(A), node(f[3])]
        a1, a2 = self.d[-1], self.d[-2]
        out = []
        for g, v, d in zip(f, vals, dead):
            g = g.clone()
            g[..., -1] = ((a2 + a1) ** 2 * g[..., -2] - a1 * a1 * g[..., -3]) / (a2 * (a2 + 2 * a1))
            g.scatter_(2, cut, v)
            out.append(torch.where(self.dead, d, g))
        Yf = torch.where(self.fuel, Y, 0.0)
        Yn = node(Yf)
        Y = torch.where((self.k == cut) & self.fuel, Yn, Y)
        return out + [torch.where(self.dead & self.fuel, 0.0, Y)[..., :self.NzY]]

    def rk(self, y):
        m = self.case["method"]
        k1 = self.phi(*y)
        if m == "Euler":
            return [a + DT * b for a, b in zip(y, k1)]
        if m == "RK2":
            k2 = self.phi(*[a + DT * b for a, b in zip(y, k1)])
            return [a + 0.5 * DT * (b + c) for a, b, c in zip(y, k1, k2)]
        k2 = self.phi(*[a + 0.5 * DT * b for a, b in zip(y, k1)])
        k3 = self.phi(*[a + 0.5 * DT * b for a, b in zip(y, k2)])
        k4 = self.phi(*[a + DT * b for a, b in zip(y, k3)])
        return [a + DT / 6 * (b + 2 * c + 2 * d + e) for a, b, c, d, e in zip(y, k1, k2, k3, k4)]

    def _solve(self, f, p):
        nx, ny, nk, d = self.Nx - 1, self.Ny - 1, self.Nz - 1, self.d
        F = torch.fft.fft(torch.fft.rfft(f[..., :nk], dim=1), dim=0)
        top = torch.fft.fft(torch.fft.rfft(p[..., -1], dim=1), dim=0)
        kx = 2 * math.pi * torch.fft.fftfreq(nx, DX, device=f.device, dtype=torch.float64)
        ky = 2 * math.pi * torch.fft.rfftfreq(ny, DX, device=f.device, dtype=torch.float64)
        kk = (kx ** 2)[:, None] + (ky ** 2)[None, :]
        sub = [0.0] + [2 / (d[q - 1] * (d[q - 1] + d[q])) for q in range(1, nk)]
        sup = [(d[0] + d[1]) / (d[0] * d[1]) - 0.5 * d[0] * kk - 1 / d[1]] + [2 / (d[q] * (d[q - 1] + d[q])) for q in range(1, nk)]
        diag = [-1.0 / d[0] * torch.ones_like(kk)] + [-(kk + 2 / (d[q - 1] * d[q])) for q in range(1, nk)]
        rhs = [0.5 * d[0] * F[..., 1]] + [F[..., q] for q in range(1, nk)]
        rhs[-1] = rhs[-1] - top / sup[-1]
        uu, yy = [diag[0]], [rhs[0]]
        for q in range(1, nk):
            l = sub[q] / uu[-1]
            uu.append(diag[q] - l * sup[q - 1])
            yy.append(rhs[q] - l * yy[-1])
        X = [None] * nk
        X[-1] = yy[-1] / uu[-1]
        for q in range(nk - 2, -1, -1):
            X[q] = (yy[q] - sup[q] * X[q + 1]) / uu[q]
        r = torch.fft.irfft(torch.fft.ifft(torch.stack(X, -1), dim=0), n=ny, dim=1)
        return torch.cat([r, p[..., -1:]], -1)

    def pressure(self, y1, yn, p):
        u, v, w, T, Y = y1
        div = self.x(u) + self.y(v) + self.zd(w)
        if not self.vardens:
            return self._solve(RHO / DT * div, p)
        Tr = T_INF * RHO
        rho = Tr / yn[3]
        Tx, Ty, Tz = self.x(T), self.y(T), self.zd(T)
        q = H_C / C_P * self._pad(Y) * self._arrhenius(T)
        dT = (12 * SIGMA_SB * DELTA * T * T * (Tx * Tx + Ty * Ty + Tz * Tz) + (K_T + 4 * SIGMA_SB * DELTA * T ** 3) * self.lap(T)) / (Tr * C_P) + q / T
        f0 = rho * (div - dT) / DT
        gr = [self.x(rho) / rho, self.y(rho) / rho, self.zd(rho) / rho]
        for _ in range(MAXIT):
            new = self._solve(f0 + gr[0] * self.x(p) + gr[1] * self.y(p) + gr[2] * self.zd(p), p)
            change = float((new - p).abs().max())
            p = new
            if change <= TOL:
                break
        return p

    def project(self, y1, yn, p):
        u, v, w, T, Y = y1
        rho = RHO * T_INF / yn[3] if self.vardens else RHO
        f = [u - DT * self.x(p) / rho, v - DT * self.y(p) / rho, w - DT * self.zd(p) / rho, T]
        Yp = torch.zeros_like(T)
        Yp[..., :self.NzY] = Y
        u, v, w, T, Y = self._walls(f, Yp, [0.0, 0.0, 0.0, T_INF])
        return [u, v, w, T.clamp(288.15, T_MAX), Y.clamp(0.0, 1.0)]

    def step(self, y, p):
        y1 = self.rk(y)
        p = self.pressure(y1, y, p)
        return self.project(y1, y, p), p


def _periodic(f):
    return torch.cat([torch.cat([f, f[:, :1]], 1), torch.cat([f[:1], f[:1, :1]], 1)], 0)


def exact(case, seed):
    dev = _device()
    out = []
    for m, size in enumerate(_sizes(case)):
        f, p = _fields(case, size, seed + 17 * m, dev)
        y, p = [a[:-1, :-1].contiguous() for a in f], p[:-1, :-1].contiguous()
        del f
        E = _Exact(case, size, seed + 17 * m if case["physics"] != "closure" else seed, dev)
        if case["kind"] == "phi":
            y, p = E.phi(*y), None
        elif case["kind"] == "rk":
            y, p = E.rk(y), None
        elif case["kind"] == "pressure":
            y, p = None, E.pressure(y, y, p)
        else:
            for _ in range(case["steps"]):
                y, p = E.step(y, p)
        r = {} if y is None else {n: _periodic(a) for n, a in zip(FIELDS, y)}
        if p is not None:
            r["p"] = _periodic(p).reshape(-1)
        out.append(r)
    return out

"""Timed workloads of the framework and their 64-bit reference results.

A case is one thing that a user's program does with the library over and over: a main-loop step
of one domain (CFL number, dt rule, TimeMarcher), a chunk of steps of a batch with its fields
brought back, some steps of a salinity run with a saved salinity frame, or one sample of the
run's statistics.  ``listed()`` gives the fixed ones, ``draw(rng)`` others of the same ranges;
``prepare`` builds the handle and writes a seeded convecting state, ``run`` makes one pass
through the public entry points, ``exact`` gives the same result from plain torch in 64 bits.

The grid tables (metrics, second-derivative coefficients, wavenumbers, interpolation stencils)
are inputs of the library's entry points: the caller owns them.  ``exact`` takes the same ones.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afid-murphfi_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import afid_gpu as ag  # noqa: E402

FIELDS = ("vx", "vy", "vz", "temp", "pr")


# ----------------------------------------------------------------------------------------------
# The cases
# ----------------------------------------------------------------------------------------------
def listed():
    return [
        # one 2-D domain, the smallest size class of a sweep: launches and the CFL readback count
        _domain("step2d_64x128_fp64", 64, 128, 1, "fp64", 1e6),
        # a test-sized 3-D domain of no special size (odd rows, lengths with factors 3 and 5)
        _domain("step3d_47x60x50_fp64", 47, 60, 50, "fp64", 1e6),
        # a mid-size 3-D run on a grid chosen by resolution, not by powers of two
        _domain("step3d_180x240x200_fp64", 180, 240, 200, "fp64", 1e8),
        # the same kind of grid in mixed precision
        _domain("step3d_225x320x300_mixed", 225, 320, 300, "mixed", 1e8),
        # the benchmark's FP64 workload
        _domain("step3d_256x384x384_fp64", 256, 384, 384, "fp64", 1e9),
        # the benchmark's mixed-precision workload, the largest case
        _domain("step3d_384x512x512_mixed", 384, 512, 512, "mixed", 1e10),
        # a parameter sweep's small class: many short columns in one batch
        _batch("sweep24_64x128_fp64", 64, 128, 1, 24, "fp64", 1e6),
        # the sweep's large class, which carries most of its cells
        _batch("sweep12_512x1024_mixed", 512, 1024, 1, 12, "mixed", 1e8),
        # a served 3-D job: a chunk of steps with the step control on the device
        _batch("job3d_96x128x128_mixed", 96, 128, 128, 1, "mixed", 1e7),
        # double-diffusive convection on two grids, refined sizes of no special ratio
        _salt("salt3d_64x72x80_r100x108x160", 64, 72, 80, 100, 108, 160, 6),
        # the documented Rayleigh-Benard example: 128^3 velocity, 384^3 scalar
        _salt("salt3d_128x128x128_r384x384x384", 128, 128, 128, 384, 384, 384, 6),
        # one sample of the statistics that a run writes at every output interval
        _stats("stats_256x192x192_fp64", 256, 192, 192, 1e8),
    ]


def _domain(name, nx, ny, nz, prec, ra):
    return _named(name, dict(kind="domain", nx=nx, ny=ny, nz=nz, prec=prec, ra=ra))


def _batch(name, nx, ny, nz, slots, prec, ra):
    # 25 steps between harvests, as the job server's benchmark runs its pools
    return _named(name, dict(kind="batch", nx=nx, ny=ny, nz=nz, slots=slots, prec=prec, ra=ra, steps=25))


def _salt(name, nx, ny, nz, nxr, nyr, nzr, steps):
    return _named(name, dict(kind="salt", nx=nx, ny=ny, nz=nz, nxr=nxr, nyr=nyr, nzr=nzr, prec="fp64", ra=1e7,
                             steps=steps))


def _stats(name, nx, ny, nz, ra):
    return _named(name, dict(kind="stats", nx=nx, ny=ny, nz=nz, prec="fp64", ra=ra))


def _named(name, case):
    if name:
        case["name"] = name
    return case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fft_len(rng, lo, hi):
    """A transform length the library takes (factors 2, 3, 5; even, as the half spectrum asks)."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    near = [n for n in range(2, 2 * hi, 2) if lo <= n <= hi and _smooth(n)]
    near.sort(key=lambda n: abs(math.log(n / want)))
    return rng.choice(near[:3])


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    kind = rng.choice(("domain2d", "domain3d", "domain3d", "domain3d", "sweep", "job3d", "salt", "stats"))
    prec = rng.choice(("fp64", "mixed"))
    if kind == "domain2d":
        return _domain(None, _log_int(rng, 40, 512), _fft_len(rng, 64, 1024), 1, prec, 1e6)
    if kind == "domain3d":
        return _domain(None, _log_int(rng, 40, 384), _fft_len(rng, 40, 480), _fft_len(rng, 40, 480), prec, 1e7)
    if kind == "sweep":
        nx, ny = _log_int(rng, 60, 512), _fft_len(rng, 100, 1024)
        return _batch(None, nx, ny, 1, max(2, min(32, _log_int(rng, 200_000, 6_000_000) // (nx * ny))), prec, 1e6)
    if kind == "job3d":
        return _batch(None, _log_int(rng, 60, 128), _fft_len(rng, 64, 144), _fft_len(rng, 64, 144), 1, prec, 1e6)
    if kind == "salt":
        nx, ny, nz = _log_int(rng, 48, 128), _fft_len(rng, 48, 128), _fft_len(rng, 48, 128)
        f = rng.uniform(1.3, 2.6)
        return _salt(None, nx, ny, nz, int(nx * f), int(ny * f), int(nz * f), 6)
    return _stats(None, _log_int(rng, 60, 300), _fft_len(rng, 64, 240), _fft_len(rng, 64, 240), 1e7)


# ----------------------------------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------------------------------
def _ratio(case):
    """Aspect ratio of the 2-D domains: a box twice as long as high."""
    return 2.0 if case["nz"] == 1 else 1.0


def _input(case, slot=0):
    """The bou.in values of the case (slot: its instance in a sweep, with a Rayleigh number of its own)."""
    i = ag.InputT()
    ra = case["ra"] * 10.0 ** (1.0 * slot / max(1, case.get("slots", 1)))
    i.nxm, i.nym, i.nzm, i.nsst = case["nx"], case["ny"], case["nz"], 3
    salt = case["kind"] == "salt"
    i.multires = i.flagsal = i.active_s = int(salt)
    i.nxmr, i.nymr, i.nzmr = case.get("nxr", i.nxm), case.get("nyr", i.nym), case.get("nzr", i.nzm)
    i.nread, i.ntst, i.walltimemax, i.tmax = 0, 10 ** 9, 1e9, 1e30
    i.tout, i.tframe, i.save_3d = 1e30, 1e30, 1e30
    i.alx3, i.ylen, i.zlen = 1.0, _ratio(case), 1.0
    # tanh-clustered walls; the two-grid runs have clipped Chebyshev velocity and uniform scalar rows
    i.istr3, i.str3, i.istr3r = (6, 12.0, 0) if salt else (4, 2.0, 4)
    i.rayt, i.prat, i.rays, i.pras, i.ffscales = ra, 1.0, (1e7 if salt else 1e8), (10.0 if salt else 1.0), int(salt)
    re = math.sqrt(ra)
    # the horizontal diffusion is explicit: dt stays below half its stability bound
    h = min(i.ylen / i.nym, i.zlen / i.nzm if i.nzm > 1 else 1e9, i.ylen / i.nymr if salt else 1e9)
    dtmax = min(1e-2, 0.5 * h * h * (math.sqrt(1e6) if salt else re))
    i.idtv, i.dt, i.resid, i.limit_cfl, i.dtmin, i.dtmax = 1, min(1e-3, dtmax, 0.3 * h), 1e-3, 1.2, 1e-12, dtmax
    i.inslws = i.inslwn = i.tfixs = i.tfixn = i.sfixs = i.sfixn = 1
    i.active_t, i.gaxis = 1, 1
    return i


def _precision(case):
    return ag.PREC_MIXED if case["prec"] == "mixed" else ag.PREC_FP64


def _modes(gen, ny, nz, dev, planes=False):
    """A smooth random y-z pattern of a few rolls, (nz, ny); planes: each z plane a pattern of its own."""
    y = torch.arange(ny, device=dev, dtype=torch.float64) * (2 * math.pi / ny)
    z = torch.arange(nz, device=dev, dtype=torch.float64) * (2 * math.pi / nz)
    r = torch.rand((6, nz if planes else 1, 4), generator=gen, dtype=torch.float64).to(dev)
    out = torch.zeros((nz, ny), device=dev, dtype=torch.float64)
    for m in range(6):
        ky = 1 + int(4 * float(r[m, 0, 0]))
        kz = 0 if planes or nz == 1 else int(4 * float(r[m, 0, 1]))
        ph = 2 * math.pi * r[m, :, 2:3]
        out += (0.2 + r[m, :, 3:4]) * torch.cos(ky * y[None, :] + kz * z[:, None] + ph)
    return out / 3.0


def _initial(case, seed, tables, dev):
    """The five fields, (nz, ny, nx + 1) with the wall row last: rolls of free-fall size in velocity and
    temperature over the conductive profile, no pressure yet.  The planes of a sweep are its instances."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 13)
    sweep = case["kind"] == "batch" and case["nz"] == 1
    ny, nz, nx = case["ny"], case["slots"] if sweep else case["nz"], case["nx"]
    xc = torch.from_numpy(tables.array("xc")).to(dev)[:nx + 1]
    xm = torch.from_numpy(tables.array("xm")).to(dev)[:nx]
    f = {n: torch.zeros((nz, ny, nx + 1), device=dev, dtype=torch.float64) for n in FIELDS}
    wx = torch.sin(math.pi * xc) ** 2
    wx[0] = wx[-1] = 0.0
    f["vx"][...] = 0.3 * _modes(gen, ny, nz, dev, sweep)[..., None] * wx
    # horizontal velocities: rolls and a weak mean shear
    f["vy"][..., :nx] = (0.3 * _modes(gen, ny, nz, dev, sweep)[..., None] + 0.05) * torch.sin(2 * math.pi * xm)
    if nz > 1 and not sweep:
        f["vz"][..., :nx] = (0.3 * _modes(gen, ny, nz, dev, sweep)[..., None] - 0.05) * torch.sin(2 * math.pi * xm)
    f["temp"][..., :nx] = 0.5 - xm + 0.1 * _modes(gen, ny, nz, dev, sweep)[..., None] * torch.sin(math.pi * xm)
    return f


def _initial_salinity(case, seed, mgrd, dev):
    gen = torch.Generator().manual_seed(int(seed) * 104729 + 29)
    x = torch.from_numpy(mgrd.array("xmr")).to(dev)[:case["nxr"]]
    return (x - 0.5) + 0.1 * _modes(gen, case["nyr"], case["nzr"], dev)[..., None] * torch.sin(math.pi * x)


class _DeviceArray:
    """A resident field as a strided device array; it keeps its owner alive."""

    def __init__(self, owner, ptr, shape, ld):
        self.owner = owner
        nz, ny, nx = shape
        self.__cuda_array_interface__ = {"shape": (nz, ny, nx), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": (ny * ld * 8, ld * 8, 8), "stream": None}


def _field(st, which):
    """Resident field `which` as a tensor (the temperature alternates between two buffers)."""
    ptr, ld = st["solver"].device_ptr(which)
    t = st["views"].get((which, ptr))
    if t is None:
        c = st["case"]
        n = c["nx"] + 1 if which == 0 else c["nx"]
        t = torch.as_tensor(_DeviceArray(st["solver"], ptr, (c["nz"], c["ny"], n), ld), device="cuda")
        st["views"][(which, ptr)] = t
    return t


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    inp = _input(case)
    tables = ag.Tables(inp, _precision(case))
    solver = ag.Solver(tables.grid, tables.params)
    st = dict(case=case, inp=inp, tables=tables, solver=solver, views={}, dt=ctypes.c_double(inp.dt), ntime=0)
    if case["kind"] == "salt":
        st["mgrd"] = ag.Mgrd(tables)
        solver.sal_create(st["mgrd"])
    f = _initial(case, seed, tables, "cuda")
    for q, n in enumerate(FIELDS):
        _field(st, q).copy_(f[n][..., :case["nx"] + 1 if q == 0 else case["nx"]])
    torch.cuda.synchronize()
    if case["kind"] == "salt":
        sal = _initial_salinity(case, seed, st["mgrd"], "cuda")
        solver.sal_upload(sal.cpu().numpy())
        # the frame goes to pinned host memory, as a program that writes it to disk keeps it
        st["frame"] = torch.empty((case["nzr"], case["nyr"], case["nxr"]), dtype=torch.float64, pin_memory=True)
    if case["kind"] != "stats":
        solver.autotune()
    solver.synchronize()
    return st


def _prepare_batch(case, seed):
    inp = _input(case)
    b = ag.Batch(inp, case["slots"], _precision(case))
    tables = ag.Tables(inp, _precision(case))
    f = {n: a.cpu().numpy() for n, a in _initial(case, seed, tables, "cuda").items()}
    for s in range(case["slots"]):
        if case["nz"] == 1:
            b.configure(s, _input(case, s))
            b.upload(s, *(f[n][s] for n in FIELDS))
        else:
            b.upload(s, *(f[n] for n in FIELDS))
    b.set_active([1] * case["slots"])
    b.autotune()
    planes = case["nz"]
    host = torch.empty((5, case["slots"] * planes, case["ny"], case["nx"] + 1), dtype=torch.float64, pin_memory=True)
    step = planes * case["ny"] * (case["nx"] + 1) * 8
    dp = ctypes.POINTER(ctypes.c_double)
    ptrs = [[ctypes.cast(host[q].data_ptr() + s * step, dp) for q in range(5)] for s in range(case["slots"])]
    return dict(case=case, batch=b, host=host, ptrs=ptrs)


# ----------------------------------------------------------------------------------------------
# One pass
# ----------------------------------------------------------------------------------------------
def _main_loop_step(st, cfl):
    err = ag.lib().afid_next_dt(ctypes.byref(st["inp"]), st["ntime"], ctypes.byref(st["dt"]), cfl, None)
    if err:
        raise RuntimeError("dt rule: %d" % err)
    st["solver"].time_marcher(st["dt"].value, st["ntime"])
    st["ntime"] += 1


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b, nx = state["batch"], case["nx"]
        b.step(case["steps"])
        for s in range(case["slots"]):
            err = ag.lib().afid_batch_download(b._h, s, *state["ptrs"][s], nx + 1, case["ny"])
            if err:
                raise RuntimeError("download: %d" % err)
        h = state["host"]
        return {n: h[q] if q == 0 else h[q][..., :nx] for q, n in enumerate(FIELDS)}
    solver = state["solver"]
    if case["kind"] == "stats":
        nu, ke, tm = solver.global_quantities(case["ra"])
        out = {"cfl": solver.calc_max_cfl(), "div": solver.check_divergence(), "nu": nu, "ke": ke, "tmean": tm}
        out.update(solver.mean_profiles())
        return out
    if case["kind"] == "salt":
        for _ in range(case["steps"]):
            cfl = solver.sal_cfl()
            _main_loop_step(state, cfl)
        fr = state["frame"]
        err = ag.lib().afid_gpu_sal_download(solver._h, ctypes.cast(fr.data_ptr(), ctypes.POINTER(ctypes.c_double)),
                                             case["nxr"], case["nyr"])
        if err:
            raise RuntimeError("sal_download: %d" % err)
        out = {n: _field(state, q) for q, n in enumerate(FIELDS)}
        out.update(sal=fr, cfl=cfl, dt=state["dt"].value)
        return out
    cfl = solver.calc_max_cfl()
    _main_loop_step(state, cfl)
    out = {n: _field(state, q) for q, n in enumerate(FIELDS)}
    out.update(cfl=cfl, dt=state["dt"].value)
    return out


def work(case):
    """Bytes and operations of one pass.  A substep cannot be merged with the next: the pressure
    couples all cells.  Per cell and substep: the fused explicit + implicit update reads five
    fields and four histories and writes four of each; the divergence is read and its half
    spectrum written; transform along z, wall-normal solve and transform back in one pass over
    it; phi written; the projection reads phi, three velocities and the pressure and writes four
    fields.  Histories, spectrum and phi are 4-byte values in mixed precision."""
    nx, ny, nz, slots = case["nx"], case["ny"], case["nz"], case.get("slots", 1)
    cells, s = nx * ny * nz * slots, 4 if case["prec"] == "mixed" else 8
    if case["kind"] == "stats":
        return {"bytes": 32 * cells, "flops": 150 * cells}
    sub = (9 * 8 + 8 * s) + (24 + s) + (2 * s if nz > 1 else 0) + 2 * s + (s + 64)
    steps = case.get("steps", 1)
    by = cells * (3 * sub + 24) * steps
    fl = cells * (3 * (260 + 5 * math.log2(ny * nz) + 60) + 8) * steps
    if case["kind"] == "batch":
        by += 40 * cells
    if case["kind"] == "salt":
        r = case["nxr"] * case["nyr"] * case["nzr"]
        by += r * (3 * (56 + 24 + 8) + 24) * steps + 8 * r  # scalar step, refined velocities, scalar read back
        fl += r * (3 * 130 + 8) * steps
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """About four times the largest difference to ``exact`` over the listed and some drawn cases.  The
    pressure sets it: the first steps of an impulsively started domain amplify rounding of the
    nearly singular mean mode by the stiff wall-normal operator (3e-10 in 64 bits, 2e-5 with
    32-bit transforms; the velocities are 1e4 to 1e6 times closer), after a chunk of steps it is
    1e-12 and 2e-6.  The statistics are plain sums."""
    if case["kind"] == "stats":
        return {"rel": 1e-13}
    first = case["kind"] == "domain"
    if case["prec"] == "mixed":
        return {"rel": 1e-4 if first else 1e-5}
    return {"rel": 1e-9 if first else 1e-11}


# ----------------------------------------------------------------------------------------------
# The same passes in plain torch, 64 bits
# ----------------------------------------------------------------------------------------------
def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = _Flow(case, seed, dev)
    if case["kind"] == "stats":
        return f.statistics(case)
    if case["kind"] == "salt":
        f.add_salinity(_Salt(case, seed, f))
    for n in range(case.get("steps", 1)):
        cfl = f.salt.cfl() if f.salt else f.cfl()
        f.next_dt(n, cfl)
        f.step()
    nx = case["nx"]
    out = {"vx": f.vx, "vy": f.vy, "vz": f.vz, "temp": f.t, "pr": f.p}
    out = {n: (a if n == "vx" else a[..., :nx]).contiguous() for n, a in out.items()}
    if case["kind"] == "batch":
        return {n: a.cpu() for n, a in out.items()}
    if f.salt:
        out["sal"] = f.salt.s.cpu()
    out.update(cfl=float(cfl), dt=float(f.dt))
    return out


def _jp(a):
    return torch.roll(a, -1, 1)


def _jm(a):
    return torch.roll(a, 1, 1)


def _tri_inverse(am, ac, ap, betadx, rows):
    """Inverses of the Crank-Nicolson matrices I - betadx d2/dx2 on `rows` (betadx: one per instance)."""
    am, ac, ap = am[rows], ac[rows], ap[rows]
    n = am.numel()
    b = betadx.reshape(-1, 1, 1)
    d2 = torch.diag(ac) + torch.diag(am[1:], -1) + torch.diag(ap[:-1], 1)
    return torch.linalg.inv(torch.eye(n, device=am.device, dtype=torch.float64) - b * d2)


class _Flow:
    def __init__(self, case, seed, dev):
        self.case, self.dev, self.salt = case, dev, None
        self.sweep = case["kind"] == "batch" and case["nz"] == 1
        self.inp = [_input(case, s) for s in range(case["slots"])] if self.sweep else [_input(case)]
        tabs = [ag.Tables(i, ag.PREC_FP64) for i in self.inp]
        tab = tabs[0]
        n = self.n = case["nx"]
        arr = lambda name, m: torch.from_numpy(tab.array(name)[:m]).to(dev)  # noqa: E731
        for a in ("udx3c", "ap3ck", "ac3ck", "am3ck", "g3rc"):
            setattr(self, a, arr(a, n + 1))
        for a in ("udx3m", "ap3sk", "ac3sk", "am3sk", "ap3ssk", "ac3ssk", "am3ssk", "amphk", "acphk", "apphk"):
            setattr(self, a, arr(a, n))
        self.xm, self.xc = tab.array("xm"), tab.array("xc")
        col = lambda v: torch.tensor(v, device=dev, dtype=torch.float64).reshape(-1, 1, 1)  # noqa: E731
        self.ren, self.pect = col([t.params.ren for t in tabs]), col([t.params.pect for t in tabs])
        self.byct = tab.params.byct
        i0 = self.inp[0]
        self.dy, self.dz, self.dx = i0.nym / i0.ylen, i0.nzm / i0.zlen, i0.nxm / i0.alx3
        nyh = i0.nym // 2 + 1
        self.ak2 = torch.stack([torch.from_numpy(t.array("ak2")[:nyh]) for t in tabs]).to(dev)[:, :, None]
        self.ak1 = torch.zeros((1, 1, 1), device=dev, dtype=torch.float64) if self.sweep else arr("ak1", i0.nzm)[:, None, None]
        f = _initial(case, seed, tab, dev)
        self.vx, self.vy, self.vz, self.t, self.p = (f[q] for q in FIELDS)
        self.dt = col([i.dt for i in self.inp])
        self.ip = (lambda a: a) if self.sweep else (lambda a: torch.roll(a, -1, 0))
        self.im = (lambda a: a) if self.sweep else (lambda a: torch.roll(a, 1, 0))

    def add_salinity(self, salt):
        self.salt = salt
        salt.interpolate(self)

    def cfl(self):
        n, vx, vy, vz = self.n, self.vx, self.vy, self.vz
        q = (((vz + self.ip(vz)) * (0.5 * self.dz)).abs() + ((vy + _jp(vy)) * (0.5 * self.dy)).abs())[..., :n]
        q = q + ((vx[..., :n] + vx[..., 1:]) * 0.5 * self.udx3m).abs()
        return (q.amax((1, 2)) if self.sweep else q.max().reshape(1)).reshape(-1, 1, 1).clamp(min=1e-8)

    def next_dt(self, ntime, cfl):
        if ntime > 1:
            top = torch.tensor([i.dtmax for i in self.inp], device=self.dev, dtype=torch.float64).reshape(-1, 1, 1)
            self.dt = torch.minimum(self.inp[0].limit_cfl / cfl, top)

    def explicit(self):
        """Advection and horizontal diffusion of vx (faces 1 .. n-1), vy, vz, temperature (rows 0 .. n-1)."""
        n, dy, dz, ip, im = self.n, self.dy, self.dz, self.ip, self.im
        vx, vy, vz, t = self.vx, self.vy, self.vz, self.t
        u, c = self.udx3m, slice(0, n)
        lap = lambda a: (_jp(a) - 2 * a + _jm(a)) * dy ** 2 + (ip(a) - 2 * a + im(a)) * dz ** 2  # noqa: E731
        avg_x = lambda a: a[..., 1:n] / u[1:] + a[..., :n - 1] / u[:-1]  # noqa: E731
        m = vx[..., 1:n]
        hx = (vx[..., 2:] + m) ** 2 - (m + vx[..., :n - 1]) ** 2
        adv = hx * 0.25
        adv = adv + 0.25 * dy * (avg_x(_jp(vy)[..., c]) * (_jp(m) + m) - avg_x(vy[..., c]) * (m + _jm(m)))
        adv = adv + 0.25 * dz * (avg_x(ip(vz)[..., c]) * (ip(m) + m) - avg_x(vz[..., c]) * (m + im(m)))
        qx = -adv * self.udx3c[1:n] + lap(m) / self.ren + self.byct * 0.5 * (t[..., 1:n] + t[..., :n - 1])

        def wall(a, shift):
            """d/dx of vx-mean times row-mean, with the wall rows repeated."""
            a = a[..., c]
            up = torch.cat((a[..., 1:], a[..., -1:]), -1) + a
            dn = a + torch.cat((a[..., :1], a[..., :-1]), -1)
            w = vx + shift(vx)
            return (w[..., 1:] * up - w[..., :n] * dn) * u * 0.25

        a = vy[..., c]
        zf = vz[..., c] + _jm(vz)[..., c]
        qy = -(wall(vy, _jm) + 0.25 * dy * ((_jp(a) + a) ** 2 - (_jm(a) + a) ** 2)
               + 0.25 * dz * ((ip(a) + a) * ip(zf) - (a + im(a)) * zf)) + lap(a) / self.ren
        b = vz[..., c]
        yf = vy[..., c] + im(vy)[..., c]
        qz = -(wall(vz, im) + 0.25 * dz * ((ip(b) + b) ** 2 - (im(b) + b) ** 2)
               + 0.25 * dy * ((_jp(b) + b) * _jp(yf) - (b + _jm(b)) * yf)) + lap(b) / self.ren
        s = t[..., c]
        up = torch.cat((s[..., 1:] + s[..., :-1], torch.full_like(s[..., :1], -1.0)), -1)   # 2 x the upper plate
        dn = torch.cat((torch.full_like(s[..., :1], 1.0), s[..., 1:] + s[..., :-1]), -1)    # 2 x the lower plate
        qt = -((vx[..., 1:] * up - vx[..., :n] * dn) * 0.5 * u
               + 0.5 * dy * (_jp(vy)[..., c] * (_jp(s) + s) - vy[..., c] * (s + _jm(s)))
               + 0.5 * dz * (ip(vz)[..., c] * (ip(s) + s) - vz[..., c] * (s + im(s)))) + lap(s) / self.pect
        if self.salt:
            qx = qx - self.salt.bycs * self.salt.salc[..., 1:]
        return qx, qy, qz, qt

    def step(self):
        n, dt = self.n, self.dt
        gam, rom = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)
        old = None
        for ns in range(3):
            ga, ro = gam[ns], rom[ns]
            al = ga + ro
            beta = dt / self.ren * 0.5
            q = self.explicit()
            if self.salt:
                self.salt.explicit()
            h = [ga * a for a in q] if old is None else [ga * a + ro * b for a, b in zip(q, old)]
            old = q
            p, c = self.p[..., :n], slice(0, n)
            v = self.vx
            d2 = v[..., 2:] * self.ap3ck[1:n] + v[..., 1:n] * self.ac3ck[1:n] + v[..., :n - 1] * self.am3ck[1:n]
            rx = (h[0] + al / self.ren * d2 - (p[..., 1:] - p[..., :-1]) * (al * self.udx3c[1:n])) * dt
            rx = rx @ _tri_inverse(self.am3ck, self.ac3ck, self.ap3ck, beta * al, slice(1, n)).transpose(1, 2)

            def d2s(a, ap, ac, am, low, up):
                """d2/dx2 with the plate values `low`, `up` (zero velocity at the walls)."""
                r = a * ac
                r[..., :-1] += a[..., 1:] * ap[:-1]
                r[..., 1:] += a[..., :-1] * am[1:]
                r[..., 0] -= (ap[0] + ac[0]) * low
                r[..., -1] -= (am[-1] + ac[-1]) * up
                return r

            inv = _tri_inverse(self.am3sk, self.ac3sk, self.ap3sk, beta * al, slice(0, n)).transpose(1, 2)
            y, z, t = self.vy[..., c], self.vz[..., c], self.t[..., c]
            # the reference's vz rows take the plain three-point sum at the walls (repeated rows)
            dz2 = z * self.ac3sk
            dz2 = dz2 + torch.cat((z[..., 1:], z[..., -1:]), -1) * self.ap3sk + torch.cat((z[..., :1], z[..., :-1]), -1) * self.am3sk
            ry = (h[1] + al / self.ren * d2s(y, self.ap3sk, self.ac3sk, self.am3sk, 0.0, 0.0)
                  - (p - _jm(p)) * (self.dy * al)) * dt
            rz = (h[2] + al / self.ren * dz2 - (p - self.im(p)) * (self.dz * al)) * dt
            rt = (h[3] + al / self.pect * d2s(t, self.ap3ssk, self.ac3ssk, self.am3ssk, 0.5, -0.5)) * dt
            ti = _tri_inverse(self.am3ssk, self.ac3ssk, self.ap3ssk, 0.5 * al * dt / self.pect, slice(0, n))
            self.vx, self.vy, self.vz, self.t = (a.clone() for a in (self.vx, self.vy, self.vz, self.t))
            self.vx[..., 1:n] += rx
            self.vx[..., 0] = self.vx[..., n] = 0.0
            self.vy[..., c] += ry @ inv
            self.vz[..., c] += rz @ inv
            self.t[..., c] += rt @ ti.transpose(1, 2)
            if self.salt:
                self.salt.implicit(ns, dt)
            self.project(al, dt, beta)
            if self.salt:
                self.salt.interpolate(self)

    def project(self, al, dt, beta):
        n, c = self.n, slice(0, self.n)
        div = ((self.ip(self.vz) - self.vz)[..., c] * self.dz + (_jp(self.vy) - self.vy)[..., c] * self.dy
               + (self.vx[..., 1:] - self.vx[..., :n]) * self.udx3m) / (al * dt)
        ny, nz = div.shape[1], div.shape[0]
        sp = torch.fft.rfft(div, dim=1)
        if not self.sweep:
            sp = torch.fft.fft(sp, dim=0)
        k2 = (self.ak2 + self.ak1)[..., 0]
        # one tridiagonal system per mode; the constant of the mean mode is fixed by phi = 0 in the last row
        mean = (k2 == 0)
        d = self.acphk[None, None, :] - k2[..., None]
        lo = self.amphk.clone()
        lo[0] = 0.0
        cp, y = [], []
        for k in range(n):
            rhs, a, b, up = sp[..., k], lo[k], d[..., k], self.apphk[k]
            if k == n - 1:
                a = torch.where(mean, torch.zeros_like(b), a.expand_as(b))
                b = torch.where(mean, torch.ones_like(b), b)
                rhs = torch.where(mean, torch.zeros_like(rhs), rhs)
            den = 1.0 / (b - a * cp[-1]) if k else 1.0 / b
            cp.append(up * den)
            y.append((rhs - a * y[-1]) * den if k else rhs * den)
        for k in range(n - 2, -1, -1):
            y[k] = y[k] - cp[k] * y[k + 1]
        sp = torch.stack(y, -1)
        del y, cp, d
        if not self.sweep:
            sp = torch.fft.ifft(sp, dim=0)
        phi = torch.fft.irfft(sp, n=ny, dim=1)
        below = torch.cat((phi[..., :1], phi[..., :-1]), -1)
        above = torch.cat((phi[..., 1:], phi[..., -1:]), -1)
        self.vx[..., c] -= (phi - below) * (al * dt * self.udx3c[:n])
        self.vy[..., c] -= (phi - _jm(phi)) * (al * dt * self.dy)
        self.vz[..., c] -= (phi - self.im(phi)) * (al * dt * self.dz)
        lap = ((self.ip(phi) - 2 * phi + self.im(phi)) * self.dz ** 2 + (_jp(phi) - 2 * phi + _jm(phi)) * self.dy ** 2
               + above * self.apphk + phi * self.acphk + below * self.amphk)
        self.p = self.p.clone()
        self.p[..., c] += phi - al * beta * lap

    def statistics(self, case):
        """The sampled numbers and y-z averaged profiles of the seeded state (no-slip walls at rest)."""
        n, c, dy, dz = self.n, slice(0, self.n), self.dy, self.dz
        ip, im = self.ip, self.im
        ren, pect = float(self.ren), float(self.pect)
        vxc, vxp = self.vx[..., :n], self.vx[..., 1:]
        vy, vz, t, vx = self.vy[..., c], self.vz[..., c], self.t[..., c], self.vx
        mean = lambda a: a.mean((0, 1)).cpu().numpy()  # noqa: E731
        xm, ym, zm = 0.5 * (vxc + vxp), 0.5 * (vy + _jp(vy)), 0.5 * (vz + ip(vz))
        w = self.g3rc[:n]
        vol = 1.0 / (self.dx * t.shape[0] * t.shape[1])
        div = (ip(vz) - vz) * dz + (_jp(vy) - vy) * dy + (vxp - vxc) * self.udx3m
        out = {"cfl": float(self.cfl()), "div": float(div.abs().max()),
               "nu": 1.0 + math.sqrt(case["ra"]) * float((t * xm * w).sum()) * vol,
               "ke": 0.5 * float(((vz ** 2 + vy ** 2 + vxc ** 2) * w).sum()) * vol, "tmean": float((t * w).sum()) * vol}
        out.update(Tbar=mean(t), vybar=mean(ym), vzbar=mean(zm), vxT=mean(xm * t), vyT=mean(ym * t), vzT=mean(zm * t),
                   Trms=np.sqrt(mean(t ** 2)), vxrms=np.sqrt(mean(0.5 * (vxc ** 2 + vxp ** 2))),
                   vyrms=np.sqrt(mean(0.5 * (vy ** 2 + _jp(vy) ** 2))), vzrms=np.sqrt(mean(0.5 * (vz ** 2 + ip(vz) ** 2))),
                   vxvy=mean(xm * ym), vxvz=mean(xm * zm), vyvz=mean(ym * zm))
        # centre metric from the cell centres, mirrored at the lower wall
        g = (self.xm[1:n + 1] - np.concatenate(([2 * self.xc[0] - self.xm[0]], self.xm[:n - 1]))) * self.dx * 0.5
        tdx = torch.from_numpy(0.5 * self.dx / g).to(self.dev)

        def ddx(a, low, up):
            """Central difference along x (two cells), with the wall values `low` and `up` at the ends."""
            r = torch.empty_like(a)
            r[..., 1:-1] = a[..., 2:] - a[..., :-2]
            r[..., 0] = a[..., 1] - a[..., 0] + 2 * (a[..., 0] - low)
            r[..., -1] = a[..., -1] - a[..., -2] + 2 * (up - a[..., -1])
            return r

        chi = ((ip(t) - im(t)) * (0.5 * dz)) ** 2 + ((_jp(t) - _jm(t)) * (0.5 * dy)) ** 2 + (ddx(t, 0.5, -0.5) * tdx) ** 2
        out["chiT"] = mean(chi) / pect
        both = lambda a: a[..., 1:] ** 2 + a[..., :n] ** 2  # noqa: E731
        yz, zy = ip(vy) - im(vy), _jp(vz) - _jm(vz)
        eps = (((ip(vz) - vz) * dz) ** 2 + ((_jp(vy) - vy) * dy) ** 2 + ((vxp - vxc) * self.udx3m) ** 2
               + 0.125 * dz ** 2 * (_jp(yz) ** 2 + yz ** 2) + 0.125 * dy ** 2 * (ip(zy) ** 2 + zy ** 2)
               + 0.125 * dz ** 2 * both(ip(vx) - im(vx)) + 0.125 * dy ** 2 * both(_jp(vx) - _jm(vx)))
        dzx, dyx = ddx(vz, 0.0, 0.0), ddx(vy, 0.0, 0.0)
        eps = eps + 0.5 * tdx ** 2 * (ip(dzx) ** 2 + dzx ** 2 + _jp(dyx) ** 2 + dyx ** 2)
        out["epsilon"] = mean(eps) / ren
        return out


class _Salt:
    """The scalar on its own grid: advection-diffusion there, the velocity brought to it by
    interpolating the three diagonal gradients and integrating them, the scalar brought back."""

    def __init__(self, case, seed, flow):
        self.mgrd = ag.Mgrd(ag.Tables(flow.inp[0], ag.PREC_FP64))
        v, dev = self.mgrd.view, flow.dev
        self.n, ny, nz = v.nxmr, v.nymr, v.nzmr
        arr = lambda p, m: torch.from_numpy(np.ctypeslib.as_array(p, shape=(m,)).copy()).to(dev)  # noqa: E731
        self.dy, self.dz, self.pecs, self.bycs = v.dyr, v.dzr, v.pecs, v.bycs
        self.ap, self.ac, self.am = (arr(p, self.n) for p in (v.ap3sskr, v.ac3sskr, v.am3sskr))
        self.u, xc = arr(v.udx3mr, self.n), arr(v.xcr, self.n + 1)
        self.lx = xc[1:] - xc[:-1]
        self.low, self.up = (arr(p, ny * nz).reshape(nz, ny) for p in (v.salbp, v.saltp))

        def stencil(s):
            return arr(s.start, s.n).long()[:, None] + torch.arange(4, device=dev), arr(s.w, 4 * s.n).reshape(-1, 4)

        self.to_ref, self.to_coarse = [stencil(s) for s in v.to_ref], [stencil(s) for s in v.to_coarse]
        self.s = _initial_salinity(case, seed, self.mgrd, dev)
        self.h = self.old = None

    @staticmethod
    def _contract(a, st, dim, wrap):
        rows, w = st
        rows = rows % a.shape[dim] if wrap else rows + 2
        shape = [1] * a.dim()
        shape[dim] = -1
        return sum(a.index_select(dim, rows[:, q].contiguous()) * w[:, q].reshape(shape) for q in range(4))

    def _interp(self, ext, st):
        return self._contract(self._contract(self._contract(ext, st[2], 0, True), st[1], 1, True), st[0], 2, False)

    @staticmethod
    def _walls(a, low, up):
        """Rows -2 .. n+1 of a column: one ghost row at each wall, zero beyond."""
        z = torch.zeros_like(a[..., :1])
        return torch.cat((z, low[..., None], a, up[..., None], z), -1)

    def interpolate(self, f):
        n, nc = self.n, f.n
        gx = (f.vx[..., 1:] - f.vx[..., :nc]) * f.udx3m
        gy = ((_jp(f.vy) - f.vy) * f.dy)[..., :nc]
        gz = ((f.ip(f.vz) - f.vz) * f.dz)[..., :nc]
        odd = lambda a: self._walls(a, -a[..., 0], -a[..., -1])  # noqa: E731
        tx = self._interp(odd(gx), self.to_ref) * self.lx
        self.vx = torch.cat((torch.zeros_like(tx[..., :1]), torch.cumsum(tx, -1)), -1)
        ty = self._interp(odd(gy), self.to_ref) / self.dy
        y0 = self._contract(self._contract(odd(f.vy[:, :1, :nc]), self.to_ref[2], 0, True), self.to_ref[0], 2, False)
        self.vy = torch.cat((y0, y0 + torch.cumsum(ty[:, :-1], 1)), 1)
        tz = self._interp(odd(gz), self.to_ref) / self.dz
        z0 = self._contract(self._contract(odd(f.vz[:1, :, :nc]), self.to_ref[1], 1, True), self.to_ref[0], 2, False)
        self.vz = torch.cat((z0, z0 + torch.cumsum(tz[:-1], 0)), 0)
        ext = self._walls(self.s, 2 * self.low - self.s[..., 0], 2 * self.up - self.s[..., -1])
        self.salc = self._interp(ext, self.to_coarse)

    def cfl(self):
        q = (((self.vz + torch.roll(self.vz, -1, 0)) * (0.5 * self.dz)).abs()
             + ((self.vy + _jp(self.vy)) * (0.5 * self.dy)).abs()
             + ((self.vx[..., :-1] + self.vx[..., 1:]) * 0.5 * self.u).abs())
        return q.max().reshape(1, 1, 1).clamp(min=1e-8)

    def explicit(self):
        s, n = self.s, self.n
        ip, im = torch.roll(s, -1, 0), torch.roll(s, 1, 0)
        mid = s[..., 1:] + s[..., :-1]
        up, dn = torch.cat((mid, 2 * self.up[..., None]), -1), torch.cat((2 * self.low[..., None], mid), -1)
        adv = (self.vx[..., 1:] * up - self.vx[..., :n] * dn) * self.u * 0.5
        adv = adv + 0.5 * self.dy * (_jp(self.vy) * (_jp(s) + s) - self.vy * (s + _jm(s)))
        adv = adv + 0.5 * self.dz * (torch.roll(self.vz, -1, 0) * (ip + s) - self.vz * (s + im))
        dif = (_jp(s) - 2 * s + _jm(s)) * self.dy ** 2 + (ip - 2 * s + im) * self.dz ** 2
        self.old, self.h = self.h, -adv + dif / self.pecs

    def implicit(self, ns, dt):
        ga, ro = ((8 / 15, 0.0), (5 / 12, -17 / 60), (3 / 4, -5 / 12))[ns]
        al, s = ga + ro, self.s
        d2 = s * self.ac
        d2[..., :-1] += s[..., 1:] * self.ap[:-1]
        d2[..., 1:] += s[..., :-1] * self.am[1:]
        d2[..., 0] -= (self.ap[0] + self.ac[0]) * self.low
        d2[..., -1] -= (self.am[-1] + self.ac[-1]) * self.up
        r = (ga * self.h + (ro * self.old if ro else 0.0) + al / self.pecs * d2) * dt
        self.s = s + r @ _tri_inverse(self.am, self.ac, self.ap, 0.5 * al * dt / self.pecs, slice(0, self.n)).transpose(1, 2)

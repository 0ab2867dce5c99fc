"""Performance cases of the FLUXOS-OVERLAND step library.

Each case is one use of the public entry points (``fluxos_cpp_b200.Domain``,
``fluxos_cpp_b200.Batch`` and ``fx_adesolver_noalloc``), from a coupler that
advances a small grid one step at a time to the 4096 x 4096 domain. The
terrains, wet starts, melt and friction fields have the distributions of
``fluxos_cpp_b200.scenarios``; they are made on the GPU from the seed, so a
large case is prepared in about a second.

Kinds of a case:

* ``step``: a domain resident on the GPU advances ``steps`` steps and its
  depth, discharges and concentrations are read back;
* ``print``: the same up to the next output time (``run_to_print``);
* ``whole``: upload of the state from the host, ``prepare``, ``steps`` steps,
  download (a coupler that owns the state);
* ``batch``: several domains of different sizes advance together;
* ``sweep``: one solute sweep on arrays that the caller owns.

A pass leaves the state advanced and the next one goes on from there (a
``whole`` or ``sweep`` pass starts from the same host or device arrays again).
Grids are indexed ``[icol, irow]`` and hold the ghost ring.
"""
import ctypes
import math

import numpy as np
import torch

import fluxos_cpp_b200 as fx

FAR = 1.0e9  # no output and no end of run within a case
ROW_TIMES = (0.0, 1.0e7, FAR, 2.0e9)  # rows of the forcing tables, from row 1
HDRY = 0.001
FILM = 0.005  # depth of the wet start [m]
SOIL_RATE = 0.5  # [1/hour]


def _case(name, kind, nr, nc, precision, steps, **more):
    c = dict(name=name, kind=kind, nr=nr, nc=nc, precision=precision, steps=steps, dxy=2, in_flight=0, terrain="fractal",
             nchem=1, ade=True, melt_field=False, manning=False, wintra=False, inflow=False, walls=False, members=1)
    c.update(more)
    return c


def listed():
    return [
        # a host model that advances this library step by step and reads the state back after each: latency and launches
        _case("couple-64", "step", 64, 64, "fp64", 1, terrain="plane"),
        # the small configuration (200 x 200 plane, uniform melt), one output interval of it
        _case("plane-200-print", "print", 200, 200, "fp64", 0, terrain="plane", print_step=90),
        # a catchment of ragged size with wall cells, in single precision, as a quick scenario run does it
        _case("catchment-257x411-fp32", "step", 257, 411, "fp32", 40, walls=True, melt_field=True, manning=True),
        # every module on: soil release, a point inflow, three solutes
        _case("modules-384", "step", 384, 384, "fp64", 20, nchem=3, wintra=True, inflow=True, melt_field=True),
        # the reference's own mode (uniform melt, no friction) on a middle-sized ragged grid
        _case("parity-1000x700", "step", 1000, 700, "fp64", 24, dxy=3),
        # dam break on a dry flat bed, two solutes
        _case("dambreak-1024-fp32", "step", 1024, 1024, "fp32", 32, terrain="dam", dxy=1, nchem=2, manning=True),
        # transport switched off in the modset: the water alone
        _case("water-only-2048-fp32", "step", 2048, 2048, "fp32", 40, ade=False, melt_field=True, manning=True),
        # a coupler that hands its grids over and takes them back around every call
        _case("whole-1024-fp32", "whole", 1024, 1024, "fp32", 20, melt_field=True, manning=True),
        # the large configuration in both precisions, as the benchmark runs it
        _case("large-4096-fp32", "step", 4096, 4096, "fp32", 63, in_flight=63, melt_field=True, manning=True),
        _case("large-4096-fp64", "step", 4096, 4096, "fp64", 20, in_flight=20, melt_field=True, manning=True),
        # an ensemble of domains of very different sizes in one batch
        _case("ensemble-12-fp32", "batch", 257, 1600, "fp32", 31, in_flight=31, members=12, manning=True),
        # the solute sweep alone on a caller's arrays
        _case("sweep-1500", "sweep", 1500, 1500, "fp64", 1, dxy=2),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "print", "whole", "batch", "sweep"])
    precision = rng.choice(["fp32", "fp64"])
    more = dict(melt_field=rng.random() < 0.5, manning=rng.random() < 0.5, dxy=rng.choice([1, 2, 3, 4, 10]))
    if kind == "step":
        nr = size(60, 3000)
        nc = max(60, min(3000, int(nr * math.exp(rng.uniform(-0.5, 0.5)))))
        c = _case("", kind, nr, nc, precision, size(1, 63), terrain=rng.choice(["fractal", "fractal", "plane"]),
                  nchem=rng.choice([1, 1, 2, 3]), ade=rng.random() < 0.85, walls=rng.random() < 0.3,
                  in_flight=rng.choice([0, 0, 8, 31]), wintra=rng.random() < 0.15, inflow=rng.random() < 0.25, **more)
        most = 3e8 / (nr * nc * (1 + c["nchem"]) * (2 if precision == "fp64" else 1))  # the large cases stay the dearest
        c["steps"] = max(1, min(c["steps"], int(most)))
    elif kind == "print":
        n = size(60, 400)
        c = _case("", kind, n, n + rng.randint(0, 60), precision, 0, terrain="plane", print_step=rng.randint(60, 240))
    elif kind == "whole":
        c = _case("", kind, size(100, 1500), size(100, 1500), precision, size(4, 40), **more)
    elif kind == "batch":
        c = _case("", kind, size(100, 300), size(400, 1400), precision, size(8, 40), members=rng.randint(4, 14), in_flight=31, **more)
    else:
        c = _case("", kind, size(60, 3000), size(60, 2500), "fp64", 1, dxy=more["dxy"])
    del c["name"]
    return c


# --- inputs -------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, lo, hi, shape):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _spectral(g, nc, nr, shape_of):
    """A random field (nc, nr) whose spectrum is shape_of(k), scaled to 0..1."""
    k = torch.hypot(torch.fft.fftfreq(nc, device="cuda")[:, None], torch.fft.rfftfreq(nr, device="cuda")[None, :]).double()
    k[0, 0] = 1.0
    amp = shape_of(k)
    amp[0, 0] = 0.0
    noise = torch.randn((2,) + tuple(k.shape), generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.irfft2(torch.complex(noise[0], noise[1]) * amp, s=(nc, nr))
    f = f - f.min()
    return f / f.max()


def _box(a):
    p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")
    return torch.nn.functional.avg_pool2d(p, 3, 1)[0, 0]


def _full(a, fill=0.0):
    g = torch.full((a.shape[0] + 2, a.shape[1] + 2), fill, dtype=a.dtype, device=a.device)
    g[1:-1, 1:-1] = a
    return g


def _extrapolate(a):
    """The ghost ring of a bed: linear from the two cells next to it."""
    a[:, 0], a[:, -1] = 1.5 * a[:, 1] - 0.5 * a[:, 2], 1.5 * a[:, -2] - 0.5 * a[:, -3]
    a[0], a[-1] = 1.5 * a[1] - 0.5 * a[2], 1.5 * a[-2] - 0.5 * a[-3]
    return a


def _grids(c, seed, nr, nc):
    """The host grids (numpy, ghost ring included) of one domain."""
    g = _generator(seed)
    dxy, n = c["dxy"], (nc, nr)
    irow = torch.arange(1, nr + 1, device="cuda", dtype=torch.float64)[None, :]
    icol = torch.arange(1, nc + 1, device="cuda", dtype=torch.float64)[:, None]
    if c["terrain"] == "plane":
        bed = 100.0 + 0.01 * (nr - irow) * dxy + _box(0.05 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    elif c["terrain"] == "dam":
        bed = torch.full(n, 10.0, device="cuda", dtype=torch.float64)
    else:
        bed = 100.0 + 3.0 * _spectral(g, nc, nr, lambda k: k ** -1.5)
        count = max(4, min(200, nr * nc // 4000))
        radius = torch.exp(_uniform(g, math.log(5.0), math.log(40.0), (count,)))
        depth, cy, cx = _uniform(g, 0.2, 1.0, (count,)), _uniform(g, 0, nr, (count,)), _uniform(g, 0, nc, (count,))
        for r, d, y, x in torch.stack([radius / dxy, depth, cy, cx], 1).tolist():  # depressions
            i, j = slice(max(0, int(x - r)), int(x + r) + 2), slice(max(0, int(y - r)), int(y + r) + 2)
            rr = torch.hypot(irow[:, j] - y, icol[i] - x)
            bed[i, j] -= torch.where(rr < r, 0.5 * d * (1.0 + torch.cos(math.pi * rr / r)), 0.0)
    bed = bed.float().double()
    if c["terrain"] == "dam":
        inside = torch.hypot(irow - 0.5 * nr, icol - 0.5 * nc) * dxy < 0.15 * min(nr, nc) * dxy * _uniform(g, 0.9, 1.1, (1,))
        h = torch.where(inside, _uniform(g, 1.95, 2.05, n), 0.0)
        conc = torch.where(inside, 1.0, 0.0)
    else:
        h = (FILM + torch.clamp(_box(_box(bed)) - bed, min=0.0)) * _uniform(g, 0.8, 1.2, n)
        conc = torch.where(h > 2 * FILM, _uniform(g, 0.5, 1.5, n), 0.0)
    wall = torch.zeros(n, device="cuda", dtype=torch.float64)
    if c["walls"]:  # NODATA areas of the DEM
        wall = (_spectral(g, nc, nr, lambda k: torch.exp(-((k * 40.0) ** 2))) > 0.8).double()
        h, conc = h * (1 - wall), conc * (1 - wall)
    zb = _extrapolate(_full(bed))
    out = {"zb": zb, "z": zb + _full(h), "h": _full(h), "qx": _full(torch.zeros_like(h)), "qy": _full(torch.zeros_like(h))}
    for k in range(c["nchem"]):
        out["conc%d" % k if k else "conc"] = _full(conc / (k + 1))
    out["ldry"], out["wall"] = _full(torch.where(h > HDRY, 0.0, 1.0)).float(), _full(wall).float()
    if c["melt_field"]:
        melt = 5.0 + 35.0 * _spectral(g, nc, nr, lambda k: torch.exp(-((k * 100.0) ** 2)))
        out["melt"] = _full(melt / melt.mean(), 1.0)
    if c["manning"]:
        out["n"] = _full(torch.full(n, 0.02, device="cuda", dtype=torch.float64) if c["terrain"] == "dam" else _uniform(g, 0.03, 0.15, n))
    if c["wintra"]:
        out["soil_mass"] = _full(_uniform(g, 0.0, 40.0, n))
    out = {k: v.cpu().numpy() for k, v in out.items()}
    out["rate"] = 0.0 if c["terrain"] == "dam" else float(_uniform(g, 5.0, 40.0, (1,)))
    return out


def _table(rate, first):
    """A forcing table: `rate` with concentration 1 until far in the future."""
    t = np.zeros((3, fx.METEO_ROWS), dtype=np.float32)
    for a, time in enumerate(ROW_TIMES):
        t[:, first + a] = (time, rate if time < FAR else 0.0, 1.0 if time < FAR else 0.0)
    return t


def _inflow_cell(nr, nc):
    return max(1, nr // 3), max(1, nc // 2)


def _d_coef(c):
    return [0.1 / (k + 1) if c["terrain"] == "dam" else 0.01 * (k + 1) for k in range(c["nchem"])]


STATE = ("zb", "z", "h", "qx", "qy")


def _solutes(c):
    return ["conc%d" % k if k else "conc" for k in range(c["nchem"])] if c["ade"] else []


def _upload(d, c, a):
    for k in STATE:
        d.upload(k, a[k])
    for k in _solutes(c) + (["soil_mass"] if c["wintra"] else []):
        d.upload(k, a[k])
    d.upload_flags(a["ldry"], a["wall"])


def _domain(c, a, nr, nc):
    d = fx.Domain(nr, nc, c["dxy"], nchem=c["nchem"], hdry=HDRY, ntim=FAR, print_step=float(c.get("print_step", FAR)),
                  ade=c["ade"], d_coef=_d_coef(c), steps_in_flight=c["in_flight"], precision=c["precision"],
                  wintra=c["wintra"], soil_release_rate=SOIL_RATE if c["wintra"] else 0.0)
    _upload(d, c, a)
    d.set_forcing(_table(a["rate"], 1))
    if "melt" in a:
        d.set_melt_field(a["melt"])
    if "n" in a:
        d.set_manning(a["n"])
    if c["inflow"]:
        d.set_inflow(_table(0.05, 0), *_inflow_cell(nr, nc))
    d.prepare()
    return d


def _wanted(c):
    return ["h", "qx", "qy"] + _solutes(c) + (["soil_mass"] if c["wintra"] else [])


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _sizes(c):
    """The members of a batch: sizes spread evenly over the logarithm, nr to nc."""
    m = c["members"]
    return [int(round(c["nr"] * (c["nc"] / c["nr"]) ** (i / max(1, m - 1)))) for i in range(m)]


def _sweep_arrays(c, seed):
    """Host grids before a solute sweep: depths, their change over the step, fluxes along the surface, flags."""
    g = _generator(seed)
    nr, nc = c["nr"], c["nc"]
    wet = _spectral(g, nc, nr, lambda k: torch.exp(-((k * 30.0) ** 2))) > 0.25
    h = torch.where(wet, _uniform(g, 0.002, 0.3, (nc, nr)), _uniform(g, 0.0, 0.0009, (nc, nr)))
    was = wet & (_uniform(g, 0, 1, (nc, nr)) > 0.02)
    q = torch.where(wet, 1.0, 0.0) * 0.05
    flags = torch.where(wet, 0, 1) | torch.where(was, 0, 2)
    return {"h": _full(h), "h0": _full(h * _uniform(g, 0.95, 1.05, (nc, nr))), "conc": _full(torch.where(wet, _uniform(g, 0, 2, (nc, nr)), 0.0)),
            "fe_1": _full(q * _uniform(g, -1, 1, (nc, nr))), "fn_1": _full(q * _uniform(g, -1, 1, (nc, nr))),
            "flags": _full(flags.to(torch.uint8), 0)}, 0.4 * c["dxy"]


def prepare(case, seed):
    c = case
    if c["kind"] == "sweep":
        a, dt = _sweep_arrays(c, seed)
        ld = (c["nr"] + 3 + 31) // 32 * 32

        def lay(v):  # the library's layout: columns padded to ld, one row of offset
            t = torch.zeros((c["nc"] + 2, ld), dtype=v.dtype, device="cuda")
            t[:, 1:c["nr"] + 3] = v
            return t

        a = {k: lay(v) for k, v in a.items()}
        a["work"] = torch.empty_like(a["conc"])
        return {"case": c, "arrays": a, "ld": ld, "dt": dt}
    if c["kind"] == "batch":
        s = {"case": c, "batch": fx.Batch(), "domains": [], "out": []}
        for i, n in enumerate(_sizes(c)):
            d = _domain(c, _grids(c, seed * 64 + i, n, n), n, n)
            s["batch"].add(d)
            s["domains"].append(d)
            s["out"].append({k: _pinned(d.shape) for k in ["h", "qx"] + _solutes(c)})
        s["batch"].set_option("steps_in_flight", c["in_flight"])
        return s
    a = _grids(c, seed, c["nr"], c["nc"])
    d = _domain(c, a, c["nr"], c["nc"])
    s = {"case": c, "domain": d, "out": {k: _pinned(d.shape) for k in _wanted(c)}}
    if c["kind"] == "whole":
        for k in list(STATE) + _solutes(c):
            p = _pinned(a[k].shape)
            p[:] = a[k]
            a[k] = p
        s["host"] = a
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "sweep":
        a = state["arrays"]
        a["work"].copy_(a["conc"])  # the host model's concentration of this step
        rc = fx.lib().fx_adesolver_noalloc(
            *(ctypes.c_void_p(a[k].data_ptr()) for k in ("work", "h", "h0", "flags", "fe_1", "fn_1")), c["nr"], c["nc"], state["ld"],
            c["dxy"], state["dt"], 0.05, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError("fx_adesolver_noalloc: %d" % rc)
        return a["work"]
    if c["kind"] == "batch":
        st = state["batch"].step(c["steps"])
        for d, out in zip(state["domains"], state["out"]):
            for k, v in out.items():
                d.download(k, v)
        return {"steps": [int(x["steps"]) for x in st], "grids": state["out"]}
    d = state["domain"]
    if c["kind"] == "whole":
        _upload(d, c, state["host"])
        d.prepare()
    if c["kind"] == "print":
        st = d.run_to_print()
        d.print_done()
    else:
        st = d.step(c["steps"])
    for k, v in state["out"].items():
        d.download(k, v)
    return {"steps": int(st["steps"]), "grids": state["out"]}


def _cells(c):
    return sum(n * n for n in _sizes(c)) if c["kind"] == "batch" else c["nr"] * c["nc"]


def work(case):
    """Bytes: each step reads and writes the state once (z, qx, qy, the solutes), reads bed, flags, friction and melt once; the
    grids that cross to the host, once. Operations: about 230 per cell of the water step and 70 per cell and solute."""
    c, n = case, _cells(case)
    if c["kind"] == "sweep":
        return {"bytes": n * (5 * 8 + 1 + 8), "flops": n * 70}
    w = 4 if c["precision"] == "fp32" else 8
    solutes = c["nchem"] if c["ade"] else 0
    steps = c["steps"] or c["print_step"]  # about a step a second
    per = 2 * w * (3 + solutes) + 8 + 1 + w * (c["manning"] + c["melt_field"]) + (2 * w * solutes if c["wintra"] else 0)
    moved = (3 if c["kind"] == "batch" else len(_wanted(c))) + (len(STATE) + solutes + 1 if c["kind"] == "whole" else 0)
    return {"bytes": n * (per * steps + 8 * moved), "flops": n * steps * (230 + 70 * solutes)}


# --- the same in 64 bits, with numpy ------------------------------------------

GACC, NUEM = float(np.float32(9.80665)), float(np.float32(1.793e-6))


def _view(a, di, dj):
    """The neighbours (icol + di, irow + dj) of the interior cells."""
    return a[1 + di:a.shape[0] - 1 + di, 1 + dj:a.shape[1] - 1 + dj]


def _upwind(hm, qn, qt, dz, dqn, dqt, dh, east):
    """The face between two wet cells: upwind part of the (mass, normal, tangential) flux and the face velocities."""
    c = np.sqrt(GACC * hm)
    u, v = qn / np.fmax(hm, HDRY), qt / np.fmax(hm, HDRY)
    cut = np.copysign(np.fmin(np.abs(dz), np.abs(dh)), dz)
    # the east face keeps a surface difference up to half the face depth
    dz = np.where(np.abs(dz) > 0.5 * hm, cut, dz) if east else cut
    cc = np.where(hm > HDRY, 0.25 / np.where(c > 0, c, 1.0), 0.0)
    a, b = u + c, u - c
    aa, ba, ua = np.abs(a), np.abs(b), np.abs(u)
    m = -((a * ba - aa * b) * dz + (aa - ba) * dqn) * cc
    n = -(a * b * (ba - aa) * dz + (aa * a - ba * b) * dqn) * cc
    t = -(v * (a * ba - 2.0 * c * ua - aa * b) * dz + v * (aa - ba) * dqn + 2.0 * c * ua * dqt) * cc
    return m, n, t, u, v


class _Numpy:
    """One domain in numpy: the step of the library in 64 bits, edge cells with the weir outflow."""

    def __init__(self, c, a, nr, nc):
        self.c, self.nr, self.nc, self.dxy = c, nr, nc, float(c["dxy"])
        for k in STATE:
            setattr(self, k, a[k].copy())
        self.dry, self.wall = a["ldry"] == 1.0, (a["wall"] == 1.0)[1:-1, 1:-1]
        self.conc = [a[k].copy() for k in _solutes(c)]
        self.soil = a["soil_mass"].copy() if c["wintra"] else None
        self.f = [np.zeros_like(self.z) for _ in range(6)]  # fe 1..3, fn 1..3
        self.rate, self.melt, self.n = float(np.float32(a["rate"])), a.get("melt"), a.get("n")
        self.tim, self.it, self.steps, self.print_next = 0.0, 0, 0, float(c.get("print_step", FAR))
        self.edge_n = np.zeros((nc, nr), bool)
        self.edge_e = np.zeros((nc, nr), bool)
        self.edge_n[[0, -1]] = True
        self.edge_e[:, [0, -1]] = True

    def step(self):
        I = (slice(1, -1), slice(1, -1))
        h, wet = self.h[I], self.h[I] > HDRY
        h0, was_dry = self.h.copy(), self.dry.copy()
        hs = np.where(wet, h, 1.0)
        speed = np.fmax(np.fmax(1e-6, np.abs(self.qx[I] / hs)), np.abs(self.qy[I] / hs)) + np.sqrt(GACC * hs)
        dt = min(self.print_next - self.tim, float(np.float32(self.dxy)) / speed[wet].max() if wet.any() else 9e10)
        self.dry[I] = ~wet
        self.tim += dt
        mi = (self.rate if self.melt is None else self.rate * self.melt[I]) / 86400000.0 * dt
        hp = np.fmax(self.z[I] - self.zb[I], 0.0)
        self.z[I] += mi
        self.h[I] = np.fmax(self.z[I] - self.zb[I], 0.0)
        self.dry[I] &= self.h[I] > HDRY
        h0[I] = self.h[I]
        had = hp != 0.0
        for k in self.conc:
            k[I] = np.where(had, (k[I] * hp + mi) / np.where(had, self.h[I], 1.0), k[I])
        if self.c["inflow"]:
            irow, icol = _inflow_cell(self.nr, self.nc)
            p = (icol, irow)
            add = float(np.float32(0.05)) * dt / (self.dxy * self.dxy)
            self.z[p] = max(self.z[p], self.zb[p])
            before = max(self.z[p] - self.zb[p], 0.0)
            self.z[p] += add
            h0[p] = self.h[p] = max(self.z[p] - self.zb[p], 0.0)
            self.dry[p] = self.h[p] <= HDRY
            for k in self.conc:
                if before != 0.0:
                    k[p] = (k[p] * before + add) / self.h[p]
        self.steps += 1
        if not wet.any():
            return
        self.it += 1
        self._water(dt)
        if self.n is not None:
            live = ~self.dry[I] & ~self.wall & (self.n[I] != 0.0)
            hh = np.where(live, self.h[I], 1.0)
            den = 1.0 + dt * GACC * self.n[I] ** 2 * np.sqrt(self.qx[I] ** 2 + self.qy[I] ** 2) / (hh * hh * np.cbrt(hh))
            self.qx[I] /= np.where(live, den, 1.0)
            self.qy[I] /= np.where(live, den, 1.0)
        if self.it > 1:
            for k, d in zip(self.conc, _d_coef(self.c)):
                _sweep(k, self.h, h0, self.dry, was_dry, self.f[0], self.f[3], self.nr, self.nc, self.dxy, dt, d)
        if self.soil is not None:
            wet = self.h[I] > HDRY
            for k in self.conc:
                out = np.where(wet, self.soil[I] * SOIL_RATE / 3600 * dt, 0.0)
                self.soil[I] -= out
                k[I] += out / (np.where(wet, self.h[I], 1.0) * self.dxy * self.dxy)

    def _water(self, dt):
        I, dxy = (slice(1, -1), slice(1, -1)), self.dxy
        self.h[I] = np.fmax(0.0, self.z[I] - self.zb[I])
        self.dry[I] = self.h[I] <= HDRY
        self.qx[I] = np.where(self.dry[I], 0.0, self.qx[I])
        self.qy[I] = np.where(self.dry[I], 0.0, self.qy[I])
        depth = np.fmax(0.0, self.z - self.zb)
        ks = np.zeros_like(self.z)
        ks[I] = HDRY
        div = np.fmax(np.fmax(depth, HDRY), ks)
        U, V = self.qx / div, self.qy / div
        zp, hp, zbp = self.z[I], depth[I], self.zb[I]
        dp, de, dn = self.dry[I], _view(self.dry, 0, 1), _view(self.dry, 1, 0)
        rough = de | dn  # a dry neighbour: no upwind part on either face
        full = np.full(zp.shape, np.inf)
        # east face, north face of the wet cells (solver_wet), and what a dry cell takes in (solver_dry)
        face = []
        for di, dj, dry_to, qn, qt in ((0, 1, de, self.qx, self.qy), (1, 0, dn, self.qy, self.qx)):
            z1, zb1 = _view(self.z, di, dj), _view(self.zb, di, dj)
            h1 = np.where(dry_to, 0.0, _view(depth, di, dj))
            q1, t1 = np.where(dry_to, 0.0, _view(qn, di, dj)), np.where(dry_to, 0.0, _view(qt, di, dj))
            over = np.fmax(0.0, zp - 0.5 * (zb1 + zbp))
            spill = over > HDRY
            dz = z1 - zp
            fall = spill & (z1 < zp)
            drop = np.where(fall, np.fmin(np.abs(dz), over), 0.0)
            cap = 0.5 * dxy * hp / dt
            weir = np.where(fall, np.fmin(0.296 * drop * np.sqrt(GACC * drop), cap), 0.0)
            hm = np.where(dry_to, np.where(spill, over, 0.0), 0.5 * (hp + h1))
            mq = np.where(dry_to, weir, 0.5 * (qn[I] + q1))
            mt = np.where(dry_to, 0.0, 0.5 * (qt[I] + t1))
            full = np.where(dry_to & fall, cap, full)
            m, n, t, u, v = _upwind(hm, mq, mt, dz, q1 - qn[I], t1 - qt[I], h1 - hp, dj == 1)
            m, n, t = (np.where(rough, 0.0, x) for x in (m, n, t))
            face.append([mq + m, mq * u + n + 0.5 * GACC * (hm * hm), mq * v + t, NUEM * np.sqrt(hp * h1)])
        vel = lambda a, di, dj: np.where(_view(self.dry, di, dj), 0.0, _view(a, di, dj))  # noqa: E731
        txe = face[0][3] * ((vel(V, 0, 1) - V[I]) / dxy + 0.25 * (vel(U, 1, 0) + _view(U, 1, 1) - _view(U, -1, 0) - _view(U, -1, 1)) / dxy)
        txn = face[1][3] * ((vel(U, 1, 0) - U[I]) / dxy + 0.25 * (vel(V, 0, 1) + _view(V, 1, 1) - _view(V, 0, -1) - _view(V, 1, -1)) / dxy)
        wet = [face[0][0], face[0][1], face[0][2] - txe, face[1][0], face[1][2] - txn, face[1][1]]
        drain = np.fmin(full, math.sqrt(GACC) * hp ** 1.5)
        wet[3] = np.where(self.edge_n, drain, wet[3])
        wet[0] = np.where(self.edge_e, drain, wet[0])
        limit = dxy * dxy * hp / dt
        e, n = wet[0] * dxy, wet[3] * dxy
        split = (wet[0] > 0) & (wet[3] > 0) & (e + n > limit)
        cf = n / np.where(split, e + n, 1.0)
        only_e, only_n = (wet[0] > 0) & ~(wet[3] > 0), (wet[3] > 0) & ~(wet[0] > 0)
        wet[0] = np.where(split, (1 - cf) * limit / dxy, np.where(only_e, np.fmin(e, limit) / dxy, wet[0]))
        wet[3] = np.where(split, cf * limit / dxy, np.where(only_n, np.fmin(n, limit) / dxy, wet[3]))
        wet[0], wet[3] = np.where(limit > 0, wet[0], 0.0), np.where(limit > 0, wet[3], 0.0)
        dry, full = [np.zeros_like(zp) for _ in range(6)], np.full(zp.shape, np.inf)
        for k, (di, dj, dry_to) in ((0, (0, 1, de)), (3, (1, 0, dn))):
            z1, h1 = _view(self.z, di, dj), _view(depth, di, dj)
            over = np.fmax(0.0, z1 - 0.5 * (_view(self.zb, di, dj) + zbp))
            live = ~dry_to & (over > HDRY)
            fall = live & (z1 > zp)
            drop = np.where(fall, np.fmin(np.abs(z1 - zp), over), 1.0)
            cap = dxy * h1 / dt
            full = np.where(fall, cap, full)
            q = -np.fmin(0.296 * drop * np.sqrt(GACC * drop), cap)
            dry[k] = np.where(fall, q, 0.0)
            dry[1 if k == 0 else 5] = np.where(fall, q * (q / (0.444 * drop)) + 0.5 * GACC * (0.444 * drop) ** 2,
                                               np.where(live, 0.5 * GACC * over * over, 0.0))
        dry[3] = np.where(self.edge_n, np.fmin(full, 0.0), dry[3])
        dry[0] = np.where(self.edge_e, np.fmin(full, 0.0), dry[0])
        stale = dp & de & dn & _view(self.dry, 0, -1) & _view(self.dry, -1, 0)
        for k in range(6):
            self.f[k][I] = np.where(self.wall, 0.0, np.where(stale, self.f[k][I], np.where(dp, dry[k], wet[k])))
        d = [((_view(self.f[k], 0, -1) - self.f[k][I]) / dxy + (_view(self.f[k + 3], -1, 0) - self.f[k + 3][I]) / dxy) * dt for k in range(3)]
        live = ~self.wall
        self.z[I] += np.where(live, d[0], 0.0)
        self.h[I] = np.fmax(0.0, self.z[I] - self.zb[I])
        out = (self.h[I] < HDRY) | self.wall
        qx = 0.1 * (_view(self.f[0], 0, -1) * dt) + 0.8 * (self.qx[I] + d[1]) + 0.1 * (self.f[0][I] * dt)
        qy = 0.1 * (_view(self.f[3], -1, 0) * dt) + 0.8 * (self.qy[I] + d[2]) + 0.1 * (self.f[3][I] * dt)
        self.qx[I], self.qy[I], self.dry[I] = np.where(out, 0.0, qx), np.where(out, 0.0, qy), out


def _sweep(c, h, h0, dry, was_dry, fe, fn, nr, nc, dxy, dt, D):
    """The solute sweep in place, anti-diagonal by anti-diagonal (cell (ix, iy) follows (ix - 1, iy) and (ix, iy - 1))."""
    I = (slice(1, -1), slice(1, -1))
    old = c.copy()
    kept = ~dry & ~was_dry
    kept[0] = kept[-1] = False
    kept[:, 0] = kept[:, -1] = False
    b = np.where(kept, c * h0 / np.where(kept, h, 1.0), c)
    b[I] = np.where(dry[I], 0.0, b[I])
    # what a cell sees on its west and south side is re-scaled already, on its east and north side not yet
    hi = np.fmax(np.fmax(_view(b, 0, -1), _view(old, 0, 1)), np.fmax(_view(b, -1, 0), _view(old, 1, 0)))
    lo = np.fmin(np.fmin(_view(b, 0, -1), _view(old, 0, 1)), np.fmin(_view(b, -1, 0), _view(old, 1, 0)))
    c[:] = b
    area = dxy * dxy
    P, flow = b[I], {}
    for name, (di, dj), q in (("e", (0, 1), fe), ("n", (1, 0), fn)):
        to, h1 = _view(b, di, dj), _view(h, di, dj)
        two = np.zeros_like(b)  # the cell after next, the ghost ring's at the edge
        if dj:
            two[:, :-2], two[:, -2:] = b[:, 2:], b[:, -1:]
            dry2 = np.concatenate([dry[:, 2:], dry[:, -1:], dry[:, -1:]], 1)
        else:
            two[:-2], two[-2:] = b[2:], b[-1:]
            dry2 = np.concatenate([dry[2:], dry[-1:], dry[-1:]], 0)
        wet = ~_view(dry, di, dj)
        disp = np.where(wet, -(np.sqrt(np.fmax(h[I] * h1, 1e-4)) / 0.5 / dxy * dxy * D) * (to - P), 0.0)
        mid = 0.5 * P + 0.5 * to
        up = wet & (q[I] > 0) & ~_view(dry, -di, -dj)
        rest = np.where(wet, np.where((q[I] > 0) | dry2[I], mid, 0.375 * P + 0.75 * to - 0.125 * two[I]), 0.0)
        edge = np.zeros_like(wet)
        edge[(slice(None), -1) if dj else (-1,)] = True
        flow[name] = [x.ravel() for x in (q[I], up, 0.75 * P, 0.375 * to, rest, edge, disp, wet, -(to * h1) * area / dt)]
    w = nr + 2
    cf, pe, pn = c.ravel(), np.zeros(c.size), np.zeros(c.size)
    store, depth, isdry = (P * h[I] * area / dt).ravel(), h[I].ravel(), dry[I].ravel()
    hi, lo = hi.ravel(), lo.ravel()
    for s in range(2, nr + nc):  # the last cell (nr, nc) is not swept
        ix = np.arange(max(1, s - nc), min(nr, s - 1) + 1)
        iy = s - ix
        at, m = iy * w + ix, (iy - 1) * nr + ix - 1
        west, south = pe[at - 1], pn[at - w]
        out = []
        for name, back in (("e", cf[at - 1]), ("n", cf[at - w])):
            q, up, p75, t375, rest, edge, disp, wet, cap = (x[m] for x in flow[name])
            f = np.where(edge, 0.0, np.fmax(0.0, np.where(up, -0.125 * back + p75 + t375, rest)))
            f = q * f * dxy + disp
            out.append(np.where(f < 0, np.where(wet, np.fmax(f, cap), 0.0), f))
        e, n = out
        have = store[m] + west + south
        split = (e > 0) & (n > 0) & (e + n > have)
        share = n / np.where(split, e + n, 1.0)
        pos = have > 0
        both = (e > 0) & (n > 0)
        e1 = np.where(split, (1 - share) * have, np.where((e > 0) & ~both, np.fmin(e, have - n), e))
        n1 = np.where(split, share * have, np.where((n > 0) & ~both, np.fmin(n, have - e), n))
        a, b2, c3 = (e >= 0) & (n < 0), (e < 0) & (n >= 0), (e >= 0) & (n >= 0)
        e2 = np.where(a, np.where(have - n > 0, np.fmin(e, have - n), 0.0), np.where(c3, 0.0, e))
        n2 = np.where(b2, np.where(have - e > 0, np.fmin(n, have - e), 0.0), np.where(c3, 0.0, n))
        e, n = np.where(pos, e1, e2), np.where(pos, n1, n2)
        d = isdry[m]
        hp = depth[m]
        new = cf[at] + (west - e + south - n) * dt / area / np.where(hp != 0, hp, 1.0)
        new = np.fmax(lo[m], np.fmin(hi[m], new))
        cf[at] = np.where(d, 0.0, new)
        pe[at], pn[at] = np.where(d, 0.0, e), np.where(d, 0.0, n)


def exact(case, seed):
    c = case
    if c["kind"] == "sweep":
        if c["nr"] + c["nc"] > 6000:
            return None
        a, dt = _sweep_arrays(c, seed)
        ld = (c["nr"] + 3 + 31) // 32 * 32
        a = {k: v.cpu().numpy() for k, v in a.items()}
        _sweep(a["conc"], a["h"], a["h0"], (a["flags"] & 1) == 1, (a["flags"] & 2) == 2, a["fe_1"], a["fn_1"], c["nr"], c["nc"], float(c["dxy"]), dt, 0.05)
        out = np.zeros((c["nc"] + 2, ld))
        out[:, 1:c["nr"] + 3] = a["conc"]
        return out
    steps = c["steps"] or c["print_step"]
    solutes = len(_solutes(c))
    if c["kind"] == "batch" or c["nr"] * c["nc"] * steps > 4e7 or solutes * (c["nr"] + c["nc"]) * steps > 90000:
        return None
    m = _Numpy(c, _grids(c, seed, c["nr"], c["nc"]), c["nr"], c["nc"])
    while (m.tim < m.print_next) if c["kind"] == "print" else (m.steps < c["steps"]):
        m.step()
    grids = {"h": m.h, "qx": m.qx, "qy": m.qy, **dict(zip(_solutes(c), m.conc))}
    if c["wintra"]:
        grids["soil_mass"] = m.soil
    return {"steps": m.steps, "grids": grids}

"""The workloads whose speed is watched: one pass of each through the library's public entry points.

A case is a plain dict.  Its "kind" names the path, the other keys its sizes and options.  Every kind
continues a simulation that the caller owns: the caller's program holds the fields on the GPU,
asks for a number of sweeps, and goes on from the buffer that the call names as the newest.

kinds
  life_bits   bit-packed GameOfLife
  life_app    the GameOfLife application's own grid (int cells, ghost ring): converted, packed,
              advanced, counted, unpacked and converted back, as a run between two outputs does
  life_u8     byte-per-cell GameOfLife
  heat        2-D heat, FP32 or FP64; with `stats` the MAX / MIN / SUM that the application prints
  himeno      Himeno pressure sweeps with gosa: plain FP32 or FP64, or FP16 defect correction
  star        radius-4 star (FDTD3d), FP32, FP16 storage or FP64, reference or weighted form
  flood       a batch of flood domains from their initial state for a number of steps
  exchange    a generic periodic stencil's ghost refresh and its three reductions
"""
import ctypes
import math

import torch

import appfis_gb300 as gb
from appfis_gb300 import _lib, workloads

DEV = "cuda"
L2_BYTES = 129e6
_TORCH = {"f32": torch.float32, "f64": torch.float64, "f16": torch.float16, "i32": torch.int32}
_CODE = {"f32": _lib.F32, "f64": _lib.F64, "f16": _lib.F16, "i32": _lib.I32}
_SIZE = {"f32": 4, "f64": 8, "f16": 2, "i32": 4}


def listed():
    return [
        # the headline GameOfLife job: fields far larger than the chip, thousands of generations
        dict(name="life_bits_16384", kind="life_bits", nx=16384, ny=16384, gens=2000, rule=0),
        # the GameOfLife application at a small size, from and to its int grid; launches and latency count
        dict(name="life_app_1024x1000", kind="life_app", nx=1024, ny=1000, gens=100, rule=0, ghost=1),
        # byte cells with rows that are no multiple of 16: the form that takes any size
        dict(name="life_u8_2050x1999", kind="life_u8", nx=2050, ny=1999, gens=20, rule=0),
        # the 2-D heat job: an L2-resident field, a thousand iterations
        dict(name="heat_1024", kind="heat", dtype="f32", nx=1024, ny=1024, pitch=1026, iters=1000, stats=False),
        # HeatDiffusion's own precision with the statistics it prints, an odd size
        dict(name="heat_f64_1000x777", kind="heat", dtype="f64", nx=1000, ny=777, pitch=1002, iters=50, stats=True),
        # Himeno's large grid, plain FP32, rows padded as the benchmark does
        dict(name="himeno_257x257x513", kind="himeno", form="f32", nx=257, ny=257, nz=513, pitch=264, iters=10, period=0, gosa=True),
        # Himeno's small grid in the reference's dense layout (rows of nx + 2)
        dict(name="himeno_dense_65x65x129", kind="himeno", form="f32", nx=65, ny=65, nz=129, pitch=67, iters=50, period=0, gosa=True),
        # the same large grid in FP16 defect correction, two periods
        dict(name="himeno_mixed_257x257x513", kind="himeno", form="mixed", nx=257, ny=257, nz=513, pitch=264, iters=40, period=20,
             gosa=True),
        # FDTD3d's large grid, weighted form
        dict(name="star_512", kind="star", dtype="f32", nx=512, ny=512, nz=512, pitch=520, iters=10, mode=1),
        # FDTD3d's reference form on an odd grid in the reference's dense layout
        dict(name="star_dense_250x127x130", kind="star", dtype="f32", nx=250, ny=127, nz=130, pitch=258, iters=10, mode=0),
        # a batch of uneven flood domains, the first steps after a dam break
        dict(name="flood_f32_6", kind="flood", dtype="f32", sides="512x700 961x624 300x1100 1325x1159 640x640 801x433", steps=20, skip_dry=False),
        # a user's own periodic stencil: what happens around its sweep
        dict(name="exchange_200x190x180", kind="exchange", dtype="f32", dims="200x190x180", ghost=1),
    ]


# ------------------------------------------------------------------------------------ drawn cases
def _sides(c):
    """(ny, nx) of every flood domain."""
    return [tuple(int(v) for v in d.split("x")) for d in c["sides"].split()]


def _cells(c):
    return sum(a * b for a, b in _sides(c))


def _dims(c):
    """Interior extents of an exchanged field, x first."""
    return [int(v) for v in c["dims"].split("x")]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _pitch(rng, width, dtype):
    """Dense rows, or rows padded to whole 32-byte sectors."""
    per = 32 // _SIZE[dtype]
    return width if rng.random() < 0.5 else -(-width // per) * per


def draw(rng):
    """A case of the listed kinds; sizes over their whole range, no larger than the largest listed."""
    kind = rng.choice(["life_bits", "life_app", "life_u8", "heat", "himeno", "himeno", "star", "star", "flood", "exchange"])
    while True:
        if kind in ("life_bits", "life_app"):
            c = dict(kind=kind, nx=32 * _log(rng, 6, 512), ny=_log(rng, 100, 16384), gens=_log(rng, 1, 2000 if kind == "life_bits" else 400),
                     rule=rng.choice([0, 0, 1]))
            if kind == "life_app":
                c["ghost"] = rng.choice([1, 1, 2])
            if c["nx"] * c["ny"] <= (1 << 28 if kind == "life_bits" else 1 << 25):
                return c
        elif kind == "life_u8":
            nx = _log(rng, 64, 8192)
            c = dict(kind=kind, nx=nx - nx % 16 if rng.random() < 0.3 else nx, ny=_log(rng, 64, 8192), gens=_log(rng, 1, 100), rule=rng.choice([0, 0, 1]))
            if c["nx"] * c["ny"] * c["gens"] <= 2e9:
                return c
        elif kind == "heat":
            dtype = rng.choice(["f32", "f32", "f64"])
            nx = _log(rng, 64, 8192)
            c = dict(kind=kind, dtype=dtype, nx=nx, ny=_log(rng, 64, 8192), pitch=_pitch(rng, nx + 2, dtype), iters=_log(rng, 1, 1000),
                     stats=rng.random() < 0.5)
            if c["nx"] * c["ny"] * c["iters"] <= (5e9 if dtype == "f32" else 5e8) and c["nx"] * c["ny"] <= 1 << 25:
                return c
        elif kind == "himeno":
            form = rng.choice(["f32", "f32", "mixed", "f64"])
            nx = _log(rng, 24, 300)
            c = dict(kind=kind, form=form, nx=nx, ny=_log(rng, 24, 300), nz=_log(rng, 24, 520), pitch=_pitch(rng, nx + 2, "f16" if form == "mixed" else "f32"),
                     iters=_log(rng, 1, 40), period=0, gosa=rng.random() < 0.7)
            if form == "mixed":
                c.update(iters=_log(rng, 10, 60), period=rng.choice([10, 20]))
            if c["nx"] * c["ny"] * c["nz"] * c["iters"] <= (1.4e9 if form != "f64" else 1.5e8):
                return c
        elif kind == "star":
            dtype = rng.choice(["f32", "f32", "f16", "f64"])
            nx = _log(rng, 20, 520)
            c = dict(kind=kind, dtype=dtype, nx=nx, ny=_log(rng, 20, 520), nz=_log(rng, 20, 520), pitch=_pitch(rng, nx + 8, dtype), iters=_log(rng, 1, 20),
                     mode=rng.choice([0, 1]))
            if c["nx"] * c["ny"] * c["nz"] * c["iters"] <= (1.4e9 if dtype != "f64" else 1.5e8):
                return c
        elif kind == "flood":
            dtype = rng.choice(["f32", "f32", "f64"])
            c = dict(kind=kind, dtype=dtype, sides=" ".join("%dx%d" % (_log(rng, 60, 1500), _log(rng, 60, 1500)) for _ in range(rng.choice([1, 1, 2, 4, 8]))),
                     steps=2 * _log(rng, 4, 40), skip_dry=rng.random() < 0.3)
            if _cells(c) * c["steps"] <= (3e8 if dtype == "f32" else 4e7):
                return c
        else:
            n = rng.choice([2, 3])
            c = dict(kind=kind, dtype=rng.choice(["f32", "f32", "f64", "i32"]), dims="x".join(str(_log(rng, 40, 4096 if n == 2 else 400)) for _ in range(n)),
                     ghost=rng.choice([1, 1, 2, 4]))
            return c


# ------------------------------------------------------------------------------------ inputs
def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + salt)


def _u(shape, seed, salt, dtype=torch.float64):
    return torch.rand(shape, generator=_gen(seed, salt), device=DEV, dtype=dtype)


def _life_cells(c, seed):
    return (_u((c["ny"], c["nx"]), seed, 1, torch.float32) < 0.3).to(torch.uint8)


def _heat_field(c, seed):
    f = torch.zeros(c["ny"] + 2, c["nx"] + 2, device=DEV, dtype=_TORCH[c["dtype"]])
    f[1:-1, 1:-1] = _u((c["ny"], c["nx"]), seed, 2, _TORCH[c["dtype"]])
    f[0] = 1.0
    return f


def _himeno_dtype(c):
    return torch.float64 if c["form"] == "f64" else torch.float32


def _himeno_fields(c, seed):
    """The benchmark's coefficients and pressure profile, each point a little off them; contractive."""
    dt, shape = _himeno_dtype(c), (c["nz"] + 2, c["ny"] + 2, c["nx"] + 2)
    coef = []
    for n in range(12):
        u = _u(shape, seed, 10 + n, torch.float32).to(dt)
        if n in (0, 1, 2, 7, 8, 9):
            coef.append(1.0 + 0.05 * (u - 0.5))
        elif n == 3:
            coef.append((0.9 + 0.05 * u) / 6.0)
        elif n in (4, 5, 6):
            coef.append(0.01 * (u - 0.5))
        else:
            coef.append(torch.ones_like(u) if n == 10 else 0.01 * u)
    p = torch.zeros(shape, device=DEV, dtype=dt)
    k = torch.arange(c["nz"], device=DEV, dtype=dt) / max(c["nz"] - 1, 1)
    p[1:-1, 1:-1, 1:-1] = (k * k)[:, None, None] + 0.01 * _u((c["nz"], c["ny"], c["nx"]), seed, 30, torch.float32).to(dt)
    return coef, p


def _star_field(c, seed):
    f = torch.zeros(c["nz"] + 8, c["ny"] + 8, c["nx"] + 8, device=DEV, dtype=_TORCH[c["dtype"]])
    f[4:-4, 4:-4, 4:-4] = (2.0 * _u((c["nz"], c["ny"], c["nx"]), seed, 3, torch.float32) - 1.0).to(f.dtype)
    return f


STAR_COEFF = 0.04  # the reference form with the mean of its 25 points: bounded over any number of steps
FLOOD = workloads.TRITON


def _flood_domains(c, seed):
    """(dem, h) per domain: a fractal bed and 1 m of water in a disc of 5% of the area."""
    doms = []
    for d, (ny, nx) in enumerate(_sides(c)):
        spec = torch.fft.rfft2(2.0 * _u((ny, nx), seed, 100 + 2 * d) - 1.0)
        k = torch.sqrt(torch.fft.fftfreq(ny, device=DEV, dtype=torch.float64)[:, None] ** 2 + torch.fft.rfftfreq(nx, device=DEV, dtype=torch.float64)[None] ** 2)
        k[0, 0] = 1.0
        spec = spec * k ** (FLOOD["beta"] / 2.0)
        spec[0, 0] = 0.0
        z = torch.fft.irfft2(spec, s=(ny, nx))
        z = z - z.min()
        z = z * (FLOOD["relief"] / z.max())
        r = math.sqrt(FLOOD["disc_area"] * nx * ny / math.pi)
        u = _u((2,), seed, 101 + 2 * d)
        cx, cy = r + u[0] * max(nx - 2 * r, 0.0), r + u[1] * max(ny - 2 * r, 0.0)
        y, x = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] + 0.5, torch.arange(nx, device=DEV, dtype=torch.float64)[None] + 0.5
        h = torch.where((x - cx) ** 2 + (y - cy) ** 2 <= r * r, FLOOD["h0"], 0.0).to(torch.float64)
        doms.append((z.contiguous(), h.contiguous()))
    return doms


def _exchange_field(c, seed):
    shape = [d + 2 * c["ghost"] for d in reversed(_dims(c))]
    u = _u(shape, seed, 4, torch.float64 if c["dtype"] == "f64" else torch.float32)
    return (u * 1000).to(torch.int32) if c["dtype"] == "i32" else u


def _rows(f, pitch):
    """The field with its rows at the pitch that the case asks for."""
    if f.shape[-1] == pitch:
        return f.clone()
    out = torch.zeros(f.shape[:-1] + (pitch,), device=DEV, dtype=f.dtype)
    out[..., : f.shape[-1]] = f
    return out


# ------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    c = dict(case)
    s = {"case": c, "cur": ctypes.c_int(0)}
    kind = c["kind"]
    if kind == "life_bits":
        cells = _life_cells(c, seed)
        a = torch.empty(c["ny"], c["nx"] // 32, device=DEV, dtype=torch.int32)
        gb.call("appfis_gb_life_pack", cells.data_ptr(), a.data_ptr(), c["nx"], c["ny"], None)
        s["buf"] = [a, torch.zeros_like(a)]
    elif kind == "life_app":
        g, nx, ny = c["ghost"], c["nx"], c["ny"]
        grid = torch.nn.functional.pad(_life_cells(c, seed).float()[None, None], (g, g, g, g), mode="circular")[0, 0].to(torch.int32)
        s["grid"] = grid.contiguous()
        s["cells"] = torch.empty(ny, nx, device=DEV, dtype=torch.uint8)
        s["buf"] = [torch.empty(ny, nx // 32, device=DEV, dtype=torch.int32) for _ in range(2)]
        s["count"] = torch.zeros(1, device=DEV, dtype=torch.int64)
    elif kind == "life_u8":
        a = _life_cells(c, seed)
        s["buf"] = [a, torch.zeros_like(a)]
    elif kind == "heat":
        a = _rows(_heat_field(c, seed), c["pitch"])
        s["buf"] = [a, a.clone()]
        s["stats"] = torch.zeros(3, device=DEV, dtype=torch.float64)
        s["box"] = (ctypes.c_int * 6)(1, c["nx"] + 1, 1, c["ny"] + 1, 0, 1)
    elif kind == "himeno":
        coef, p = _himeno_fields(c, seed)
        coef = [_rows(f, c["pitch"]) for f in coef]
        a = _rows(p, c["pitch"])
        s.update(coef=coef, ptrs=(ctypes.c_void_p * 12)(*[f.data_ptr() for f in coef]), buf=[a, a.clone()])
        if c["form"] == "mixed":
            s["half"] = torch.empty(13 * a.numel(), device=DEV, dtype=torch.float16)
        s["gosa"] = torch.zeros(c["iters"], device=DEV, dtype=torch.float64) if c["gosa"] else None
    elif kind == "star":
        a = _rows(_star_field(c, seed), c["pitch"])
        s["buf"] = [a, a.clone()]
        s["w"] = ((ctypes.c_double if c["dtype"] == "f64" else ctypes.c_float) * 5)(*workloads.fdtd_weights()) if c["mode"] == 1 else None
    elif kind == "flood":
        s["doms"] = _flood_domains(c, seed)
        n, dt = len(s["doms"]), _TORCH[c["dtype"]]
        s["table"] = (_lib.FloodDomain * n)()
        s["fields"] = []
        for d, (ny, nx) in enumerate(_sides(c)):
            pitch = -(-(nx + 2) // 32) * 32
            f = torch.zeros(8, ny + 2, pitch, device=DEV, dtype=dt)  # h, qx, qy twice each, dem, n2
            s["fields"].append(f)
            t = s["table"][d]
            t.nx, t.ny, t.pitch = nx, ny, pitch
            for k in range(2):
                t.h[k], t.qx[k], t.qy[k] = f[k].data_ptr(), f[2 + k].data_ptr(), f[4 + k].data_ptr()
            t.dem, t.n2 = f[6].data_ptr(), f[7].data_ptr()
        s["prm"] = _lib.FloodParams(FLOOD["dx"], FLOOD["courant"], FLOOD["hextra"], FLOOD["t_end"], FLOOD["t_end"], FLOOD["time_step"], 0.0, c["steps"],
                                    _lib.FLOOD_SKIP_DRY if c["skip_dry"] else 0)
        s["steps"] = torch.zeros(n, device=DEV, dtype=torch.int32)
    else:
        s["field"] = _exchange_field(c, seed)
        dims = [d + 2 * c["ghost"] for d in _dims(c)]
        s["dims"] = (ctypes.c_int * len(dims))(*dims)
        box = []
        for d in _dims(c):
            box += [c["ghost"], c["ghost"] + d]
        s["box"] = (ctypes.c_int * 6)(*(box + [0, 1] * (3 - len(dims))))
        s["result"] = torch.zeros(3, device=DEV, dtype=torch.int64 if c["dtype"] == "i32" else torch.float64)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------ run
def _newest(s):
    """Puts the buffer that the call left the newest state in first."""
    if s["cur"].value:
        s["buf"].reverse()


def _reduce(field, code, px, py, box, out, k):
    gb.call("appfis_gb_reduce", field.data_ptr(), code, px, py, box, k, out.data_ptr() + 8 * k, None)


def run(state):
    s, c = state, state["case"]
    kind, cur = c["kind"], ctypes.byref(state["cur"])
    if kind == "life_bits":
        a, b = s["buf"]
        gb.call("appfis_gb_life_bits", a.data_ptr(), b.data_ptr(), c["nx"], c["ny"], c["gens"], c["rule"], cur, None)
        _newest(s)
        return list(s["buf"])
    if kind == "life_app":
        nx, ny, g, grid, cells, (a, b) = c["nx"], c["ny"], c["ghost"], s["grid"], s["cells"], s["buf"]
        gb.call("appfis_gb_life_from_i32", grid.data_ptr(), nx + 2 * g, g, cells.data_ptr(), nx, ny, None)
        gb.call("appfis_gb_life_pack", cells.data_ptr(), a.data_ptr(), nx, ny, None)
        b.zero_()
        gb.call("appfis_gb_life_bits", a.data_ptr(), b.data_ptr(), nx, ny, c["gens"], c["rule"], cur, None)
        _newest(s)
        a = s["buf"][0]
        gb.call("appfis_gb_life_population_bits", a.data_ptr(), a.numel(), s["count"].data_ptr(), None)
        gb.call("appfis_gb_life_unpack", a.data_ptr(), cells.data_ptr(), nx, ny, None)
        gb.call("appfis_gb_life_to_i32", cells.data_ptr(), nx, ny, grid.data_ptr(), nx + 2 * g, g, None)
        return {"grid": grid, "population": s["count"]}
    if kind == "life_u8":
        a, b = s["buf"]
        gb.call("appfis_gb_life_u8", a.data_ptr(), b.data_ptr(), c["nx"], c["ny"], c["gens"], c["rule"], cur, None)
        _newest(s)
        return list(s["buf"])
    if kind == "heat":
        a, b = s["buf"]
        gb.call("appfis_gb_heat2d" if c["dtype"] == "f32" else "appfis_gb_heat2d_f64", a.data_ptr(), b.data_ptr(), c["nx"], c["ny"], c["pitch"],
                c["iters"], 0.2, 0.2, cur, None)
        _newest(s)
        if c["stats"]:
            for k in range(3):
                _reduce(s["buf"][0], _CODE[c["dtype"]], c["pitch"], c["ny"] + 2, s["box"], s["stats"], k)
        return {"field": s["buf"][0][:, : c["nx"] + 2], "stats": s["stats"]}
    if kind == "himeno":
        (a, b), gosa = s["buf"], s["gosa"].data_ptr() if c["gosa"] else None
        if c["form"] == "mixed":
            gb.call("appfis_gb_himeno_mixed", s["ptrs"], a.data_ptr(), b.data_ptr(), s["half"].data_ptr(), c["nx"], c["ny"], c["nz"], c["pitch"],
                    c["iters"], c["period"], 0.8, gosa, cur, None)
        else:
            gb.call("appfis_gb_himeno" if c["form"] == "f32" else "appfis_gb_himeno_f64", s["ptrs"], a.data_ptr(), b.data_ptr(), c["nx"], c["ny"],
                    c["nz"], c["pitch"], c["iters"], 0.8, gosa, cur, None)
        _newest(s)
        out = {"p": s["buf"][0][:, :, : c["nx"] + 2]}
        if c["gosa"]:
            out["gosa"] = s["gosa"]
        return out
    if kind == "star":
        a, b = s["buf"]
        if c["dtype"] == "f64":
            gb.call("appfis_gb_star_r4_f64", a.data_ptr(), b.data_ptr(), c["nx"], c["ny"], c["nz"], c["pitch"], c["iters"], c["mode"], STAR_COEFF,
                    s["w"], cur, None)
        else:
            gb.call("appfis_gb_star_r4", a.data_ptr(), b.data_ptr(), _CODE[c["dtype"]], c["nx"], c["ny"], c["nz"], c["pitch"], c["iters"], c["mode"],
                    STAR_COEFF, s["w"], _lib.STAR_AUTO, 0, cur, None)
        _newest(s)
        return s["buf"][0][:, :, : c["nx"] + 8]
    if kind == "flood":
        code = _CODE[c["dtype"]]
        for t, (dem, h) in zip(s["table"], s["doms"]):
            gb.call("appfis_gb_flood_setup", ctypes.byref(t), code, dem.data_ptr(), h.data_ptr(), None, None, FLOOD["manning"], None)
        gb.call("appfis_gb_flood_run", s["table"], len(s["doms"]), code, ctypes.byref(s["prm"]), None, s["steps"].data_ptr(), None, None, None)
        # an even number of steps, well before t_end: the newest state is in the first buffers
        return {"steps": s["steps"], "fields": [[f[k][:, : t.nx + 2] for k in (0, 2, 4)] for f, t in zip(s["fields"], s["table"])]}
    gb.call("appfis_gb_ghost_periodic", s["field"].data_ptr(), _SIZE[c["dtype"]], len(s["dims"]), s["dims"], c["ghost"], None)
    for k in range(3):
        _reduce(s["field"], _CODE[c["dtype"]], s["dims"][0], s["dims"][1], s["box"], s["result"], k)
    return {"field": s["field"], "result": s["result"]}


# ------------------------------------------------------------------------------------ work
def _traffic(resident, per_sweep, sweeps):
    """Bytes of a run of sweeps: a field that fits on the chip crosses the memory once for all of
    them, a larger one once for each."""
    return per_sweep * (sweeps if resident > L2_BYTES else 1)


def work(case):
    """Bytes and operations that one pass cannot do without.  Integer logic counts as one operation
    per 32-bit word, as the machine does it."""
    c, kind = case, case["kind"]
    if kind in ("life_bits", "life_app", "life_u8"):
        n = c["nx"] * c["ny"]
        cell = 1.0 if kind == "life_u8" else 0.125
        b = _traffic(2 * cell * n, 3 * cell * n, c["gens"])
        if kind == "life_bits":
            b = 4 * cell * n  # two states in, two out: any number of generations can be blocked on chip
        if kind == "life_app":
            b = 2.0 * 4 * (c["nx"] + 2 * c["ghost"]) * (c["ny"] + 2 * c["ghost"])
        return {"bytes": b, "flops": 11.0 * n / 32 * c["gens"]}
    if kind == "heat":
        n, e = c["nx"] * c["ny"], _SIZE[c["dtype"]]
        return {"bytes": _traffic(2.0 * e * n, 2.0 * e * n, c["iters"]), "flops": 9.0 * n * c["iters"]}
    if kind == "himeno":
        n = c["nx"] * c["ny"] * c["nz"]
        per = {"f32": 56.0, "f64": 112.0, "mixed": 30.0}[c["form"]]
        return {"bytes": _traffic(per * n, per * n, c["iters"]), "flops": 34.0 * n * c["iters"]}
    if kind == "star":
        n, e = c["nx"] * c["ny"] * c["nz"], _SIZE[c["dtype"]]
        return {"bytes": _traffic(2.0 * e * n, 2.0 * e * n, c["iters"]), "flops": (25.0 if c["mode"] == 0 else 29.0) * n * c["iters"]}
    if kind == "flood":
        n, e = _cells(c), _SIZE[c["dtype"]]
        # the FP64 initial state in, then bed, roughness and state read and state written per step
        return {"bytes": 16.0 * n + _traffic(8.0 * e * n, 8.0 * e * n, c["steps"]), "flops": 10.0 * n * c["steps"]}
    n, e = math.prod(_dims(c)), _SIZE[c["dtype"]]
    padded = math.prod(d + 2 * c["ghost"] for d in _dims(c))
    return {"bytes": float(e) * (n + 2 * (padded - n)), "flops": 3.0 * n}


# ------------------------------------------------------------------------------------ exact
def _life_exact(c, cells):
    cur, old = cells, torch.zeros_like(cells)
    one, zero = torch.ones_like(cells), torch.zeros_like(cells)
    for _ in range(c["gens"]):
        rows = cur + torch.roll(cur, 1, 1) + torch.roll(cur, -1, 1)
        n = rows + torch.roll(rows, 1, 0) + torch.roll(rows, -1, 0) - cur
        if c["rule"] == 0:
            new = torch.where(cur == 1, torch.where((n < 2) | (n > 4), zero, old), torch.where(n == 3, one, old))
        else:
            new = torch.where(cur == 1, (n == 2) | (n == 3), n == 3).to(torch.uint8)
        cur, old = new, cur
    return cur, old


def _pack(cells):
    w = cells.reshape(cells.shape[0], -1, 32)
    out = torch.zeros(w.shape[:2], device=DEV, dtype=torch.int64)
    for k in range(32):
        out |= w[:, :, k].to(torch.int64) << k
    return torch.where(out >= 1 << 31, out - (1 << 32), out).to(torch.int32)


def _himeno_exact(c, seed):
    coef, p = _himeno_fields(c, seed)
    a0, a1, a2, a3, b0, b1, b2, c0, c1, c2, bnd, w1 = [f.double()[1:-1, 1:-1, 1:-1] for f in coef]
    del coef
    p = p.double()
    gosa = torch.zeros(c["iters"], device=DEV, dtype=torch.float64)
    nz, ny, nx = c["nz"], c["ny"], c["nx"]

    def at(dx, dy, dz):
        return p[1 + dz:1 + dz + nz, 1 + dy:1 + dy + ny, 1 + dx:1 + dx + nx]

    for it in range(c["iters"]):
        s0 = a0 * at(1, 0, 0) + a1 * at(0, 1, 0) + a2 * at(0, 0, 1)
        s0 += b0 * (at(1, 1, 0) - at(1, -1, 0) - at(-1, 1, 0) + at(-1, -1, 0))
        s0 += b1 * (at(0, 1, 1) - at(0, -1, 1) - at(0, 1, -1) + at(0, -1, -1))
        s0 += b2 * (at(1, 0, 1) - at(-1, 0, 1) - at(1, 0, -1) + at(-1, 0, -1))
        s0 += c0 * at(-1, 0, 0) + c1 * at(0, -1, 0) + c2 * at(0, 0, -1) + w1
        ss = (s0 * a3 - at(0, 0, 0)) * bnd
        gosa[it] = (ss * ss).sum()
        p = p.clone()
        p[1:-1, 1:-1, 1:-1] += 0.8 * ss
    return {"p": p, "gosa": gosa} if c["gosa"] else {"p": p}


def _star_exact(c, seed):
    f = _star_field(c, seed).double()
    nz, ny, nx = c["nz"], c["ny"], c["nx"]
    w = workloads.fdtd_weights()

    def at(dx, dy, dz):
        return f[4 + dz:4 + dz + nz, 4 + dy:4 + dy + ny, 4 + dx:4 + dx + nx]

    for _ in range(c["iters"]):
        v = at(0, 0, 0) * (1.0 if c["mode"] == 0 else w[0])
        for a in range(1, 5):
            ring = at(-a, 0, 0) + at(a, 0, 0) + at(0, -a, 0) + at(0, a, 0) + at(0, 0, -a) + at(0, 0, a)
            v = v + ring * (1.0 if c["mode"] == 0 else w[a])
        f[4:-4, 4:-4, 4:-4] = v * (STAR_COEFF if c["mode"] == 0 else 1.0)
    return f


def _face(a, b, nx, ny, dx, dt, hextra, D):
    """Contributions of the faces between cells a and b (h, qx, qy, z each) to a and to b."""
    G, SG, E = 9.81, 3.132091953, 1e-12
    (h1, p1, q1, z1), (h2, p2, q2, z2) = a, b
    zero = torch.zeros_like(h1)
    wet = (h1 > 0) | (h2 > 0)

    def ratio(n, d, ok):
        return torch.where(ok, n / torch.where(ok, d, torch.ones_like(d)), zero)

    u1, v1 = ratio(p1, h1, h1 >= hextra), ratio(q1, h1, h1 >= hextra)
    u2, v2 = ratio(p2, h2, h2 >= hextra), ratio(q2, h2, h2 >= hextra)
    s1, s2 = torch.sqrt(h1.clamp(min=0)), torch.sqrt(h2.clamp(min=0))
    dh, c12 = h2 - h1, torch.sqrt(G * 0.5 * (h1 + h2))
    u12, v12 = ratio(u1 * s1 + u2 * s2, s1 + s2, wet), ratio(v1 * s1 + v2 * s2, s1 + s2, wet)
    un = u12 * nx + v12 * ny
    l0, l1, l2 = un - c12, un, un + c12
    n1, n2 = u1 * nx + v1 * ny, u2 * nx + v2 * ny
    e1, e2 = n1 - SG * s1, n2 - SG * s2
    fix = (e1 < 0) & (e2 > 0)
    t = ratio(e1 * (e2 - l0), e2 - e1, fix)
    le0, l0 = torch.where(fix, l0 - t, zero), torch.where(fix, t, l0)
    e1, e2 = n1 + SG * s1, n2 + SG * s2
    fix = (e1 < 0) & (e2 > 0)
    t = ratio(e2 * (l2 - e1), e2 - e1, fix)
    le2, l2 = torch.where(fix, l2 - t, zero), torch.where(fix, t, l2)
    dp, dq = p2 - p1, q2 - q1
    m = ratio((dp * nx + dq * ny) - un * dh, c12, wet)
    al0, al2 = 0.5 * (dh - m), 0.5 * (dh + m)
    al1 = ratio((dq - v12 * dh) * nx - (dp - u12 * dh) * ny, c12, wet)
    dz = z2 - z1
    up = dz >= 0
    dzp = torch.where(up, torch.where(z1 + h1 < z2, h1, dz), torch.where(z2 + h2 < z1, -h2, dz))
    be = ratio(0.5 * G * (torch.where(up, h1, h2) - 0.5 * dzp.abs()) * dzp, c12, wet)
    hp = h1 + al0
    sub = (l0 * l2 < 0) & (hp > 0) & (h1 > 0) & (h2 > 0)
    lim = torch.minimum(torch.maximum(be, al0 * l0 - h1 * dx * 0.5 / dt), -al2 * l2 + h2 * dx * 0.5 / dt)
    be = torch.where(sub, lim, be)
    w0, w1, w2 = l0 * al0 - be, l1 * al1, l2 * al2 + be
    right = (hp - be / l2 < -D) & (h2 < D)
    left = ~right & (hp - be / l0 < -D) & (h1 < D)
    plain = ~right & ~left
    waves = [(l0, w0, 1.0, u12 - c12 * nx, v12 - c12 * ny, plain), (l1, w1, 0.0, -c12 * ny, c12 * nx, plain),
             (l2, w2, 1.0, u12 + c12 * nx, v12 + c12 * ny, plain), (le0, le0 * al0, 1.0, u12 - c12 * nx, v12 - c12 * ny, wet),
             (le2, le2 * al2, 1.0, u12 + c12 * nx, v12 + c12 * ny, wet)]
    d1, d2 = [torch.where(right, w0 + w2, zero), zero, zero], [torch.where(left, w0 + w2, zero), zero, zero]
    for lam, w, r0, r1, r2, on in waves:
        for k, r in enumerate((r0, r1, r2)):
            d2[k] = d2[k] + torch.where(on & (lam > 0), w * r, zero)
            d1[k] = d1[k] + torch.where(on & ~(lam > 0), w * r, zero)
    out = []
    for d in (d1, d2):
        out.append([torch.where(wet & (x.abs() >= E), dt * x / dx, zero) for x in d])
    return out


def _flood_exact(c, seed):
    """The batch in 64 bits; None for FP32 fields after more than 20 steps: a cell whose depth rounds
    across a wet/dry threshold takes another branch, and after that many steps the two precisions
    follow different fronts."""
    steps = torch.full((len(_sides(c)),), c["steps"], device=DEV, dtype=torch.int32)
    if c["dtype"] == "f32" and c["steps"] > 20:
        return {"steps": steps, "fields": [[None] * 3 for _ in _sides(c)]}
    # the depth below which a cell counts as dry is part of each form's definition
    dx, hextra, E, D = FLOOD["dx"], FLOOD["hextra"], 1e-12, 1e-12 if c["dtype"] == "f64" else 1e-6
    fields = []
    for dem, h0 in _flood_domains(c, seed):
        dem, h0 = dem.to(_TORCH[c["dtype"]]).double(), h0.to(_TORCH[c["dtype"]]).double()
        pad = torch.nn.functional.pad
        z = pad(dem, (1, 1, 1, 1), value=1e6)
        h = pad(h0, (1, 1, 1, 1))
        p, q = torch.zeros_like(h), torch.zeros_like(h)
        for _ in range(c["steps"]):
            hi, pi, qi = h[1:-1, 1:-1], p[1:-1, 1:-1], q[1:-1, 1:-1]
            safe, root = torch.where(hi > hextra, hi, torch.ones_like(hi)), torch.sqrt(9.81 * hi)
            cfl = torch.minimum(dx / ((pi / safe).abs() + root), dx / ((qi / safe).abs() + root)) * FLOOD["courant"]
            cfl = torch.where(hi > hextra, cfl, torch.full_like(cfl, math.inf)).min()
            dt = torch.where(torch.isinf(cfl), torch.full_like(cfl, FLOOD["time_step"]), cfl)
            cells = lambda y, x: tuple(f[y, x] for f in (h, p, q, z))  # noqa: E731
            r = [torch.zeros_like(h) for _ in range(6)]
            y, x = slice(1, -1), slice(1, -1)
            lo, hi_ = slice(None, -1), slice(1, None)
            fa, fb = _face(cells(y, lo), cells(y, hi_), 1.0, 0.0, dx, dt, hextra, D)
            for k in range(3):
                r[k][y, lo] += fa[k]
                r[3 + k][y, hi_] += fb[k]
            fa, fb = _face(cells(hi_, x), cells(lo, x), 0.0, 1.0, dx, dt, hextra, D)
            for k in range(3):
                r[k][hi_, x] += fa[k]
                r[3 + k][lo, x] += fb[k]
            hn = hi
            new = (hn - r[0][y, x] - r[3][y, x]).clamp(min=0)
            mx, my = pi - r[1][y, x] - r[4][y, x], qi - r[2][y, x] - r[5][y, x]
            mod, nn = torch.sqrt(mx * mx + my * my), FLOOD["manning"] ** 2
            rub = (hn >= hextra) & (mod > E)
            tt = dt * 9.81 * nn * mod / (torch.where(rub, hn, torch.ones_like(hn)) ** (7.0 / 3.0))
            den = torch.where(rub, 0.5 * (1.0 + torch.sqrt(1.0 + 4.0 * tt)), torch.ones_like(tt))
            dry = new < hextra
            mx, my = torch.where(dry, torch.zeros_like(mx), mx / den), torch.where(dry, torch.zeros_like(my), my / den)
            h, p, q = pad(new, (1, 1, 1, 1)), pad(mx, (1, 1, 1, 1)), pad(my, (1, 1, 1, 1))
            level = new + z[y, x]

            def blocked(dy, dx_):
                s = (slice(1 + dy, h.shape[0] - 1 + dy), slice(1 + dx_, h.shape[1] - 1 + dx_))
                return (level < z[s]) & (h[s] < D)

            wet = new > hextra
            p[y, x] = torch.where(wet & (blocked(0, 1) | blocked(0, -1)), torch.zeros_like(mx), mx)
            q[y, x] = torch.where(wet & (blocked(-1, 0) | blocked(1, 0)), torch.zeros_like(my), my)
        fields.append([h, p, q])
    return {"steps": steps, "fields": fields}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("life_bits", "life_u8", "life_app"):
        if c["nx"] * c["ny"] * c["gens"] > 6e11:
            return None
        cur, old = _life_exact(c, _life_cells(c, seed))
        if kind == "life_u8":
            return [cur, old]
        if kind == "life_bits":
            return [_pack(cur), _pack(old)]
        g = c["ghost"]
        grid = torch.nn.functional.pad(cur.float()[None, None], (g, g, g, g), mode="circular")[0, 0].to(torch.int32)
        return {"grid": grid, "population": cur.sum(dtype=torch.int64).reshape(1)}
    if kind == "heat":
        f = _heat_field(c, seed).double()
        for _ in range(c["iters"]):
            v = f[1:-1, 1:-1]
            f[1:-1, 1:-1] = v + 0.2 * (f[1:-1, :-2] + f[1:-1, 2:] - 2 * v) + 0.2 * (f[:-2, 1:-1] + f[2:, 1:-1] - 2 * v)
        v = f[1:-1, 1:-1]
        stats = torch.stack([v.max(), v.min(), v.sum()]) if c["stats"] else torch.zeros(3, device=DEV, dtype=torch.float64)
        return {"field": f, "stats": stats}
    if kind == "himeno":
        return _himeno_exact(c, seed)
    if kind == "star":
        return _star_exact(c, seed)
    if kind == "flood":
        return _flood_exact(c, seed)
    f, g = _exchange_field(c, seed), c["ghost"]
    for axis in range(f.dim() - 1, -1, -1):
        n = f.shape[axis]
        f.narrow(axis, 0, g).copy_(f.narrow(axis, n - 2 * g, g).clone())
        f.narrow(axis, n - g, g).copy_(f.narrow(axis, g, g).clone())
    v = f[tuple(slice(g, -g) for _ in range(f.dim()))]
    v = v.to(torch.int64 if c["dtype"] == "i32" else torch.float64)
    return {"field": f if c["dtype"] == "i32" else f.double(), "result": torch.stack([v.max(), v.min(), v.sum()])}

"""The work that programs have this library do, as measurable cases.

A case is one pass of a kind of program:

  run       a segment of an LES run between two field outputs: the stored field
            goes to the device (lesgpu_set_fields, as a restart with IREAD = 1
            does), the time loop takes `steps` steps and reads each step's
            report (lesgpu_step), and the fields come back (lesgpu_get_fields)
            into the program's pinned buffers.  With `averages` the run also
            accumulates field_avg's statistics and writes them.  The mixed
            form holds its velocities and temperature to about single precision, so a
            program that uses it passes its fields on in single precision on
            the GPU; the FP64 form's stay as they are.
  poisson   one allocation-free pressure solve on device buffers
            (lesgpu_poisson_ftft_noalloc), as a plugin calls it.
  serving   a few immersed-body cases submitted together to a running server
            and read back as they finish.

Flows of `run` (field `flow`):
  channel   turbulent channel with heat transfer, periodic x and z, FFT Poisson
  duct      the channel closed by walls in z, x FFT + multigrid (poiss_x_ft)
  mgrd      the channel solved by BiCGSTAB + 3-D multigrid (poiss_mgrd)
  body      flow past a heated body: convective outlet, immersed boundary, z
            FFT + x-y multigrid (poiss_z_ft); `conjugate` conducts heat in it
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import time

import numpy as np
import torch

import leswht_gb300
from leswht_gb300 import abi, cases, ibmpre, serving
from leswht_gb300.gridgen import axis_vectors

FIELDS = ("u", "v", "w", "p", "t")
BODY = {"cylinder": abi.BODY_CYLINDER, "square": abi.BODY_SQUARE, "sphere": abi.BODY_SPHERE}


def _run(name, flow, n1, n2, n3, form, steps, **kw):
    c = {"name": name, "kind": "run", "flow": flow, "n1": n1, "n2": n2, "n3": n3, "form": form, "steps": steps}
    c.update(kw)
    return c


def listed():
    return [
        # a plugin's pressure solve: a small ragged grid, where the launches are the cost ...
        {"name": "poisson_30x33x24", "kind": "poisson", "n1": 30, "n2": 33, "n3": 24},
        # ... and about the largest that fits the entry point's fixed scratch
        {"name": "poisson_128x125x120", "kind": "poisson", "n1": 128, "n2": 125, "n3": 120},
        # the Re_tau = 180 channel, both forms: the everyday size
        _run("channel_64_mixed", "channel", 64, 64, 64, "mixed", 10),
        _run("channel_64_fp64", "channel", 64, 64, 64, "fp64", 6),
        # a ragged channel whose run collects the time averages of its statistics
        _run("channel_90x81x96_fp64_averages", "channel", 90, 81, 96, "fp64", 3, averages=True),
        # the Re_tau = 590 channel, the largest resident case
        _run("channel_384x256x384_mixed", "channel", 384, 256, 384, "mixed", 3),
        # bodies in a free stream: a small one in FP64, where launches count ...
        _run("body_64x48x8_fp64", "body", 64, 48, 8, "fp64", 4, body="cylinder", re=100.0),
        # ... the Re = 100 cylinder, and the Re = 3900 cylinder
        _run("body_128x96x16_mixed", "body", 128, 96, 16, "mixed", 6, body="cylinder", re=100.0),
        _run("body_256x192x64_mixed", "body", 256, 192, 64, "mixed", 3, body="cylinder", re=3900.0),
        # a square duct: walls in y and z, the other FFT + multigrid solver
        _run("duct_64x48x48_mixed", "duct", 64, 48, 48, "mixed", 4),
        # the third pressure solver, on a small channel
        _run("mgrd_32x32x32_fp64", "mgrd", 32, 32, 32, "fp64", 2),
        # the serving loop: five bodies of uneven sizes on the GPU at once
        {"name": "serving_5x30_mixed", "kind": "serving", "count": 5, "largest": 4, "steps": 30},
    ]


def _smooth(rng, lo, hi, step=1):
    """A length the transforms take (2^p 3^q 5^r), log-uniform in [lo, hi]."""
    ok = []
    for n in range(lo, hi + 1):
        m = n
        for q in (2, 3, 5):
            while m % q == 0:
                m //= q
        if m == 1 and n % step == 0:
            ok.append(n)
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(ok, key=lambda n: abs(n - x))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("poisson", "channel", "body", "duct", "mgrd", "serving"), (3, 5, 5, 2, 1, 1))[0]
    if kind == "poisson":
        while True:
            c = {"kind": "poisson", "n1": _smooth(rng, 16, 128), "n2": _log(rng, 17, 128), "n3": _smooth(rng, 16, 128)}
            if 24 * c["n1"] * (c["n3"] // 2 + 1) * c["n2"] < (31 << 20):
                return c
    if kind == "serving":
        return {"kind": "serving", "count": rng.randint(2, 5), "largest": rng.randint(1, 4), "steps": rng.randint(10, 30)}
    form = rng.choice(("mixed", "fp64"))
    c = {"kind": "run", "flow": kind, "form": form}
    if kind == "channel":
        while True:
            c.update(n1=_smooth(rng, 24, 256), n2=_log(rng, 24, 192), n3=_smooth(rng, 24, 256))
            if c["n1"] * c["n2"] * c["n3"] <= (6e6 if form == "mixed" else 1.5e6):
                break
        c.update(steps=rng.randint(2, 5), averages=rng.random() < 0.25)
    elif kind == "duct":
        c.update(n1=_smooth(rng, 24, 96), n2=_log(rng, 24, 64), n3=16 * rng.randint(2, 4), steps=rng.randint(2, 4))
    elif kind == "mgrd":
        c.update(n1=rng.choice((16, 32, 64)), n2=_log(rng, 24, 64), n3=rng.choice((16, 32, 64)), steps=1)
    else:
        while True:
            c.update(n1=32 * rng.randint(2, 8), n2=_log(rng, 48, 192), n3=_smooth(rng, 4, 64))
            if c["n1"] * c["n2"] * c["n3"] <= (3.2e6 if form == "mixed" else 4e5):
                break
        c.update(body=rng.choice(sorted(BODY)), re=float(_log(rng, 40, 3900)), steps=rng.randint(2, 4),
                 conjugate=rng.random() < 0.2)
    return c


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=2)
def _base(flow, n1, n2, n3, form, body, re, averages, conjugate):
    """The unperturbed case: settings, grid, pre-processor tables, base flow."""
    prec = abi.PREC_MIXED if form == "mixed" else abi.PREC_FP64
    if flow == "body":
        case = cases.cylinder(n1, n2, n3, re=re, body_kind=BODY[body], amp=0.0, precision=prec)
        if conjugate:
            s = dict(case.settings, iconjg=1)
            axes = axis_vectors(case.grid_dat, False, False, True)
            cs, ks, om = ibmpre.conjg_tables_gpu(leswht_gb300.load_library(), s, case.grid, axes, 2.0, 5.0)
            case.settings = s
            case.ibm = dict(case.ibm, cstar=cs, kstar=ks, omega=om)
    else:
        box = dict(lx=2 * math.pi, lz=math.pi, re=10950.0) if n1 * n2 * n3 > 2 ** 22 else {}
        if flow == "duct":
            box = dict(lx=2 * math.pi, lz=2.0, zwalls=True)
        case = cases.channel(n1, n2, n3, amp=0.0, precision=prec, **box)
        case.ibm = None                  # no body: the library's unit tables
        if flow == "duct":
            nlev = 0
            while nlev < 4 and n3 % (2 ** (nlev + 1)) == 0 and n3 // (2 ** (nlev + 1)) >= 2:
                nlev += 1
            case = cases.with_poisson(case, abi.POISSON_X_FT, nlev)
        elif flow == "mgrd":
            case = cases.with_poisson(case, abi.POISSON_MGRD)
        if averages:
            case.settings = dict(case.settings, iavg=1, avg_tst=-1.0)
    case.ihist, case.m = 0, 0
    return case


def _perturbed(case, seed, amp):
    """The base flow with a uniform perturbation of relative amplitude `amp` on
    the interior unknowns, as prefld leaves it (periodic ghost copies), in
    pinned host memory."""
    s, g = case.settings, case.grid
    n1, n2, n3, n1m, n2m, n3m = g.n1, g.n2, g.n3, g.n1m, g.n2m, g.n3m
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    f = {k: torch.from_numpy(case.fields[k]).cuda() for k in FIELDS}
    wall = 1 if s["zprdic"] == 1 else 2
    inside = {"u": (slice(1, n3), slice(1, n2), slice(1 if s["xprdic"] == 1 else 2, n1)),
              "v": (slice(1, n3), slice(2, n2), slice(1, n1)),
              "w": (slice(wall, n3), slice(1, n2), slice(1, n1))}
    solid = f["u"] == 0.0
    area = {"u": (torch.from_numpy(g.f2fz)[:, None, None], torch.from_numpy(g.f2fy)[None, :, None], 2),
            "v": (torch.from_numpy(g.f2fz)[:, None, None], torch.from_numpy(g.f2fx)[None, None, :], 1),
            "w": (torch.from_numpy(g.f2fy)[None, :, None], torch.from_numpy(g.f2fx)[None, None, :], 0)}
    for k in ("u", "v", "w"):
        r = torch.rand(f[k].shape, generator=gen, dtype=torch.float64, device="cuda").sub_(0.5).mul_(2.0 * amp)
        keep = torch.zeros_like(r)
        keep[inside[k]] = 1.0
        r *= keep
        if s["ich"] == 1:                # a closed channel: no net flux of the perturbation through any plane
            a, b, normal = area[k]
            over = [d for d in range(3) if d != normal]
            wgt = keep * a.cuda() * b.cuda()
            r -= keep * ((r * wgt).sum(over, keepdim=True) / wgt.sum(over, keepdim=True).clamp_min(1e-300))
        elif k == "u":
            r.masked_fill_(solid, 0.0)
        f[k] += r
    if s["ich"] == 1:                    # the decomposed temperature follows the flow, t = u / Pr
        c = (slice(1, n3), slice(1, n2), slice(1, n1))
        e = (slice(1, n3), slice(1, n2), slice(2, n1 + 1))
        f["u"][:, :, n1] = f["u"][:, :, 1]
        f["t"][c] = 0.5 * (f["u"][c] + f["u"][e]) / s["pr"]
    if s["xprdic"] == 1:
        for k in ("u", "v", "w", "t"):
            f[k][:, :, 0] = f[k][:, :, n1m]
            f[k][:, :, n1] = f[k][:, :, 1]
    if s["zprdic"] == 1:
        for k in ("u", "v", "w", "t"):
            f[k][0] = f[k][n3m]
            f[k][n3] = f[k][1]
    out = {}
    for k in FIELDS:
        out[k] = torch.empty(f[k].shape, dtype=torch.float64, pin_memory=True)
        out[k].copy_(f[k])
    return out


def _case_base(c):
    return _base(c["flow"], c["n1"], c["n2"], c["n3"], c["form"], c.get("body"), c.get("re"), c.get("averages", False),
                 c.get("conjugate", False))


SERVED = (((64, 48, 8), "square", 60.0), ((96, 64, 16), "cylinder", 100.0), ((128, 96, 16), "sphere", 400.0),
          ((96, 64, 16), "square", 250.0), ((192, 128, 32), "cylinder", 900.0))


@functools.lru_cache(maxsize=None)
def _uniform_grid(n1, n2, n3):
    case = cases.channel(n1, n2, n3, amp=0.0)
    return case.grid, abi.pack_grid(case.grid)


def prepare(case, seed):
    if case["kind"] == "poisson":
        lib = leswht_gb300.load_library()
        fn = lib.lesgpu_poisson_ftft_noalloc
        fn.argtypes = [C.POINTER(abi.Grid), C.c_void_p, C.c_void_p, C.c_void_p]
        fn.restype = C.c_int
        g, packed = _uniform_grid(case["n1"], case["n2"], case["n3"])
        return {"kind": "poisson", "fn": fn, "grid": packed, "div": _divergence(g, seed),
                "phi": torch.zeros(g.shape, dtype=torch.float64, device="cuda")}
    if case["kind"] == "serving":
        batch = []
        for q in range(case["count"]):
            (n1, n2, n3), body, re = SERVED[min(case["largest"], q)]
            b = _served_base(n1, n2, n3, body, re)
            f = _perturbed(b, seed * 16 + q, 1.0e-3)
            batch.append(cases.Case(b.name, b.settings, b.grid, b.grid_dat, b.grid_bin, {k: f[k].numpy() for k in FIELDS},
                                    time=b.time, dt=b.dt, ibm=b.ibm))
        return {"kind": "serving", "batch": batch, "steps": case["steps"],
                "server": serving.Server(leswht_gb300.load_library(), max_active=8)}
    base = _case_base(case)
    f = _perturbed(base, seed, 1.0e-3 if case["flow"] == "body" else 0.1)
    host = {k: f[k].numpy() for k in FIELDS}
    solver = leswht_gb300.gpu_solver(cases.Case(base.name, base.settings, base.grid, base.grid_dat, base.grid_bin, host,
                                                time=base.time, dt=base.dt, ibm=base.ibm))
    out = {k: torch.empty(f[k].shape, dtype=torch.float64, pin_memory=True) for k in FIELDS}
    return {"kind": "run", "solver": solver, "host": host, "dt": base.dt, "out": out, "steps": case["steps"],
            "mixed": case["form"] == "mixed", "averages": case.get("averages", False)}


@functools.lru_cache(maxsize=None)
def _served_base(n1, n2, n3, body, re):
    return cases.cylinder(n1, n2, n3, re=re, body_kind=BODY[body], amp=0.0, precision=abi.PREC_MIXED)


def _divergence(g, seed):
    """A right-hand side with the solvability of a divergence: no net source."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    d = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    inner = torch.randn((g.n3m, g.n2m, g.n1m), generator=gen, dtype=torch.float64, device="cuda")
    wy = torch.from_numpy(g.f2fy[1:g.n2m + 1]).cuda()[None, :, None]
    inner -= (inner * wy).sum() / (wy.sum() * g.n1m * g.n3m)
    d[1:g.n3m + 1, 1:g.n2m + 1, 1:g.n1m + 1] = inner
    return d


# --------------------------------------------------------------------- run
REPORTED = ("time", "dt", "ubulk", "tbulk_fluid", "csgsts", "qflux")


def run(state):
    if state["kind"] == "poisson":
        stream = torch.cuda.current_stream().cuda_stream
        rc = state["fn"](C.byref(state["grid"].struct), state["div"].data_ptr(), state["phi"].data_ptr(), stream)
        if rc != 0:
            raise RuntimeError(f"lesgpu_poisson_ftft_noalloc: {abi.ERR_NAMES.get(rc, rc)}")
        return state["phi"]
    if state["kind"] == "serving":
        server = state["server"]
        waiting = [server.submit(c, state["steps"]) for c in state["batch"]]
        results = {}
        while len(results) < len(waiting):
            for n, ticket in enumerate(waiting):
                if n not in results and server.poll(ticket)[0] >= serving.DONE:
                    fields, _, _ = server.result(ticket)
                    server.release(ticket)
                    results[n] = {k: _single(torch.from_numpy(fields[k])) for k in FIELDS}
            time.sleep(2.0e-4)
        return [results[n] for n in range(len(waiting))]
    solver = state["solver"]
    solver.set_fields(state["host"], 0.0, state["dt"], 0, 0)
    for _ in range(state["steps"]):
        report = solver.step()
    out = state["out"]
    ptr = [C.cast(out[k].data_ptr(), abi.PD) for k in FIELDS]
    rc = solver.lib.lesgpu_get_fields(solver.h, *ptr)
    if rc != 0:
        raise RuntimeError(f"lesgpu_get_fields: {abi.ERR_NAMES.get(rc, rc)}")
    result = {k: _single(out[k]) if state["mixed"] else out[k] for k in FIELDS}
    scalars = [report[k] for k in REPORTED] + report["cd"][:1]
    result["report"] = np.array(scalars, np.float32 if state["mixed"] else np.float64)
    if state["averages"]:
        sums, result["samples"] = solver.averages(reset=True)
        result["averages"] = {k: _single(torch.from_numpy(v)) if state["mixed"] else v for k, v in sums.items()}
    return result


def _single(a):
    return a.to("cuda", non_blocking=True).to(torch.float32)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: what the step's phases cannot do without at the widths the form
    stores (each operand once per phase: 289 words a cell and step in FP64,
    236 word equivalents in the mixed form, as bench.py counts them; bodies
    about as much), the fields' transfers, and the statistics' sums.  A solve
    reads the right-hand side and writes phi.  Operations: about 1300 a cell
    and step (stencils 450, SGS 500, sweeps 250, transforms 100)."""
    if case["kind"] == "poisson":
        cells = case["n1"] * case["n2"] * case["n3"]
        return {"bytes": 16.0 * cells, "flops": cells * (2.5 * 2 * math.log2(case["n1"] * case["n3"]) + 9)}
    if case["kind"] == "serving":
        cells = sum(math.prod(SERVED[min(case["largest"], q)][0]) for q in range(case["count"]))
        words, steps = 236, case["steps"]
    else:
        cells = case["n1"] * case["n2"] * case["n3"]
        words, steps = (236 if case["form"] == "mixed" else 289), case["steps"]
    b = cells * (8.0 * words * steps + 80.0)
    if case.get("averages"):
        b += cells * 23 * 8.0 * (2 * steps + 1)
    return {"bytes": b, "flops": 1300.0 * cells * steps}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The pressure solve in 64 bits with plain torch: FFT in x and z, the y
    systems by elimination; the mean mode's last row is replaced by phi = 0 and
    the mode shifted so that the replaced row holds.  A whole step has no such
    value here."""
    if case["kind"] != "poisson":
        return None
    g, _ = _uniform_grid(case["n1"], case["n2"], case["n3"])
    div = _divergence(g, seed)
    n1m, n2m, n3m = g.n1m, g.n2m, g.n3m
    rhs = torch.fft.fft(torch.fft.rfft(div[1:n3m + 1, 1:n2m + 1, 1:n1m + 1], dim=0), dim=2).transpose(0, 1)
    kx = 2.0 * (1.0 - torch.cos(2.0 * math.pi * torch.arange(n1m, dtype=torch.float64) / n1m)) * g.f2fxi[1] ** 2
    kz = 2.0 * (1.0 - torch.cos(2.0 * math.pi * torch.arange(n3m // 2 + 1, dtype=torch.float64) / n3m)) * g.f2fzi[1] ** 2
    k2 = (kz[:, None] + kx[None, :]).cuda()
    lower = [0.0] + [g.f2fyi[j] * g.c2cyi[j] for j in range(2, n2m + 1)]
    upper = [g.f2fyi[j] * g.c2cyi[j + 1] for j in range(1, n2m)] + [0.0]
    x, gam = [], []
    prev_x = prev_g = None
    for j in range(n2m):
        diag, b, up, lo = -(lower[j] + upper[j] + k2), rhs[j].clone(), torch.full_like(k2, upper[j]), torch.full_like(k2, lower[j])
        if j == n2m - 1:
            diag[0, 0], lo[0, 0], b[0, 0] = 1.0, 0.0, 0.0
        if j > 0:
            diag = diag - lo * prev_g
            b = b - lo * prev_x
        prev_g, prev_x = up / diag, b / diag
        gam.append(prev_g)
        x.append(prev_x)
    for j in range(n2m - 2, -1, -1):
        x[j] = x[j] - gam[j] * x[j + 1]
    shift = (rhs[n2m - 1][0, 0] - lower[n2m - 1] * x[n2m - 2][0, 0]) / -(lower[n2m - 1] + upper[n2m - 1])
    for j in range(n2m - 1):
        x[j][0, 0] -= shift
    phi = torch.fft.irfft(torch.fft.ifft(torch.stack(x).transpose(0, 1), dim=2), n=n3m, dim=0)
    out = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    out[1:n3m + 1, 1:n2m + 1, 1:n1m + 1] = phi
    return out

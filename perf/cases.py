"""Performance cases of the framework: what its users have it do, through its
public entry points, with the sizes of its configurations, tests and benchmark.

Three kinds of case:
  solve   frehd_cg_solve_noalloc on device arrays the caller owns
  domain  one domain advanced by `steps` time steps and its state read back:
          `frehd_domain_run`, or step by step with the statistics of every step
          (a host that steers the model); FP64 or mixed, geometry from the fine
          bottoms or from level tables, one or more scalars, with or without TVD
          advection, inflow and wind
  batch   an ensemble admitted into a batch, stepped together, released and
          read back
  served  the same ensemble submitted to the continuous-batching server, each
          request with its own step count

Every pass goes on from where the last one ended, as a model run does.  Inputs
come from the seed: a smooth random bed with 4 x 4 fine pixels per cell, dry
land, a sine tide on the north row, a small initial wave and scalar plumes.
"""
import math

import numpy as np
import torch

from frehdc_b200 import native

G = 9.81
R = 4                       # fine pixels per cell edge
SERIES = 1 << 15            # entries of the forcing series (steps a domain may run)
BUDGET = 24 << 30           # device bytes a batch or server may hold
FIELDS = ["surf", "uuXP", "vvYP", "S"]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest call: the solve of a host that owns its device memory, on a
        # basin of the test decks' size; latency only.
        _solve("solve_48x40", 48, 40),
        # The same entry at its largest size.
        _solve("solve_512x512", 512, 512),
        # A host that steers the model step by step and reads every step's
        # statistics, on a small odd grid.
        _domain("stepwise_117x93", 117, 93, 10, stepwise=True),
        # The 128 x 128 basin of the parity runs, one output interval per pass.
        _domain("basin_128x128", 128, 128, 20),
        # Ragged basin from level tables with TVD advection, an inflow and wind.
        _domain("forced_tables_301x187", 301, 187, 10, geometry="tables", adv=2, forced=True),
        # The 512 x 512 window of the large estuary, with two scalars.
        _domain("window_512x512", 512, 512, 20, dx=2.0, dt=0.5, dry=0.3, scalars=2),
        # A mid-size estuary whose sides fit no tile.
        _domain("estuary_1500x1003", 1500, 1003, 12, dx=2.0, dt=0.5, dry=0.3),
        # The large estuary in FP64: the headline workload.
        _domain("estuary_4096x4096", 4096, 4096, 16, dx=2.0, dt=0.5, dry=0.3),
        # A large domain in mixed precision.
        _domain("mixed_2048x2048", 2048, 2048, 20, dx=2.0, dt=0.5, dry=0.3, precision="mixed"),
        # A small one in mixed precision, 1:4.
        _domain("mixed_160x640", 160, 640, 16, precision="mixed", scalars=2),
        # An ensemble of uneven basins in mixed precision, two scalars each.
        _group("ensemble_24_mixed", "batch", 24, 64, 512, 30, "mixed", 65536.0),
        # Requests of uneven size and length served together.
        _group("served_12_fp64", "served", 12, 64, 256, 24, "fp64", 16384.0),
    ]


def _solve(name, nx, ny):
    return {"name": name, "kind": "solve", "nx": nx, "ny": ny}


def _domain(name, nx, ny, steps, dx=10.0, dt=1.0, dry=0.2, precision="fp64", geometry="fine",
            scalars=1, adv=1, forced=False, stepwise=False):
    return {"name": name, "kind": "domain", "nx": nx, "ny": ny, "steps": steps, "dx": dx, "dt": dt,
            "dry": dry, "precision": precision, "geometry": geometry, "scalars": scalars,
            "adv": adv, "forced": forced, "stepwise": stepwise}


def _group(name, kind, count, smin, smax, steps, precision, cells_per_cta):
    return {"name": name, "kind": kind, "count": count, "smin": smin, "smax": smax,
            "steps": steps, "precision": precision, "cells_per_cta": cells_per_cta}


def draw(rng):
    """Another case of the same ranges."""
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["solve", "domain", "domain", "domain", "domain", "batch", "served"])
    if kind == "solve":
        return _unnamed(_solve("", side(24, 512), side(24, 512)))
    if kind == "domain":
        fine_dx = rng.random() < 0.5
        nx, ny = side(40, 2400), side(40, 2400)
        tables = nx * ny <= 60000 and rng.random() < 0.4
        return _unnamed(_domain(
            "", nx, ny, rng.randint(6, 20), dx=2.0 if fine_dx else 10.0,
            dt=0.5 if fine_dx else 1.0, dry=rng.choice([0.1, 0.2, 0.3]),
            precision=rng.choice(["fp64", "fp64", "mixed"]),
            geometry="tables" if tables else "fine", scalars=rng.randint(1, 3),
            adv=rng.choice([1, 1, 2]), forced=rng.random() < 0.25, stepwise=rng.random() < 0.25))
    return _unnamed(_group("", kind, rng.randint(6, 24), 64, side(128, 512), rng.randint(10, 30),
                           rng.choice(["fp64", "mixed"]), float(rng.choice([16384, 65536, 131072]))))


def _unnamed(case):
    del case["name"]
    return case


# ------------------------------------------------------------------ inputs
def _rng(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _min_rows(z, ny, nx):
    """Per cell: the minimum over y of each of its R pixel columns, (ny, nx, R)."""
    return z.view(ny, R, nx, R).amin(1)


def _deck(nx, ny, seed, dx=10.0, dt=1.0, dry=0.2, scalars=1, adv=1, forced=False, amp=0.3,
          manning=0.025, depth=5.0):
    """Inputs of one domain (device tensors, deck datum)."""
    g = _rng(seed, 1)
    f64 = dict(dtype=torch.float64, device="cuda")
    w = torch.randn(ny, nx, generator=g, **f64)
    corr = min(200.0, 0.2 * dx * min(nx, ny))  # correlation length of the bed, m
    ky, kx = torch.fft.fftfreq(ny, dx, **f64), torch.fft.rfftfreq(nx, dx, **f64)
    filt = torch.exp(-2.0 * (math.pi * corr) ** 2 * (ky[:, None] ** 2 + kx ** 2))
    f = torch.fft.irfft2(torch.fft.rfft2(w) * filt, s=(ny, nx))
    f = (f - f.min()) / (f.max() - f.min())
    # about `dry` of the bed above low tide; open water at the tidal (north) row
    some = f.flatten()[:: max(1, nx * ny // 200000)].sort().values
    high = some[min(len(some) - 1, int((1.0 - dry) * len(some)))] if dry > 0 else 1.3
    z = -depth + (depth - amp) / high * f
    xb = (ny - torch.arange(ny, **f64) - 0.5) * dx
    t = (xb / (0.08 * ny * dx)).clamp(max=1.0)
    cap = torch.where(t < 1.0, -(amp + 1.0) * (1.0 - t) ** 2, torch.full_like(t, math.inf))
    z = torch.minimum(z + 1e-4 * xb[:, None], cap[:, None])
    zf = torch.nn.functional.interpolate(z[None, None], scale_factor=R, mode="bilinear",
                                         align_corners=False)[0, 0]
    zf += 0.4 * torch.rand(ny * R, nx * R, generator=g, **f64) - 0.2
    cols, rows = _min_rows(zf, ny, nx), zf.view(ny, R, nx, R).amin(3)
    bx, by = cols[:, :, R - 1].clone(), rows[:, R - 1, :].clone()
    bx[:, :-1] = torch.maximum(bx[:, :-1], cols[:, 1:, 0])
    by[:-1] = torch.maximum(by[:-1], rows[1:, 0, :])
    surf = (0.05 * torch.sin(2.0 * math.pi * xb / (ny * dx)))[:, None].expand(ny, nx).contiguous()
    x = (torch.arange(nx, **f64) + 0.5 - 0.5 * nx) * dx
    y = (torch.arange(ny, **f64) + 0.5 - 0.5 * ny) * dx
    sig = 0.1 * dx * min(nx, ny)
    S = []
    for s in range(scalars):
        a = 2.0 * math.pi * s / max(scalars, 1)
        off = 0.25 * dx * (0 if s == 0 else min(nx, ny))
        S.append((1.0 - 0.2 * s) * torch.exp(-((x - off * math.cos(a)) ** 2 +
                                               ((y - off * math.sin(a)) ** 2)[:, None]) / (2 * sig ** 2)))
    bottom = cols.amin(2)
    steps = np.arange(SERIES)
    d = {"zf": zf, "bottom": bottom, "bxp": bx, "byp": by, "surf": surf, "S": S,
         "tide": amp * np.sin(2.0 * math.pi * steps * dt / 44712.0)}
    i0, j0 = nx // 3, ny // 3
    inflow = (i0, i0 + 3, j0, j0 + 2) if forced else (0, 0, 0, 0)
    smax = round(max(amp, 0.05) + 0.05, 6)
    d["cfg"] = dict(
        nx=nx, ny=ny, dx=dx, dy=dx, dt=dt, g=G, NUx=1e-4, NUy=1e-4, Kx=1e-4, Ky=1e-4, CDx=0.01,
        CDy=0.01, manningN=manning, CDmax=1.0, hD=0.1, CwT=10.0, CDnotN=0, useThinLayer=1,
        useSubgrid=1, useSubDrag=0, staggeredV=1, useminA=0, useminV=3, dxf=dx / R, dyf=dx / R,
        subR=float(R), surfmin=-smax, surfmax=smax, dsurf=0.01, bcType=1, tideLocFirstP=0,
        tideLocLengthP=nx, useScalar=1, scalarAdv=adv, useConstTidePS=1, tidePS=0.0,
        useWind=int(forced), useEvap=0, useRain=0, inflowLocLength=6 if forced else 0,
        useSubStep=0, checkConservation=0, minDepth=1e-5, wtfh=1e-5, CFLl=0.5, CFLh=0.7, eps=1e-12,
        maxIter=100000, offset=float(-bottom.min()), inflowI0=inflow[0], inflowI1=inflow[1],
        inflowJ0=inflow[2], inflowJ1=inflow[3], inflowS=1.0, northAngle=15.0, rhoa=1.25, Cw=0.0013,
        nscalar=scalars)
    if forced:
        ph = 2.0 * math.pi * steps * dt / 10800.0
        d["series"] = {native.SERIES_INFLOW: 3.0 * (1.0 + 0.5 * np.sin(ph)),
                       native.SERIES_WIND_SPEED: 7.0 * (1.0 + 0.3 * np.sin(ph)),
                       native.SERIES_WIND_DIR: 60.0 + 20.0 * np.sin(0.7 * ph)}
    return d


def _case_deck(case, seed):
    return _deck(case["nx"], case["ny"], seed, case["dx"], case["dt"], case["dry"], case["scalars"],
                 case["adv"], case["forced"])


def _members(case, seed):
    """Size, steps and deck parameters of an ensemble's basins.  The sizes are the
    case's own (whatever the seed): spread over [smin, smax], square or 1:4."""
    out = []
    n = case["count"]
    for k in range(n):
        a = case["smin"] * (case["smax"] / case["smin"]) ** (k / max(n - 1, 1))
        nx, ny = (a, a) if k % 2 == 0 else (a / 2, a * 2)
        steps = case["steps"] if case["kind"] == "batch" else max(1, case["steps"] * (1 + k % 4) // 4)
        out.append((max(8, round(nx)), max(8, round(ny)), steps, int(seed) * 64 + k,
                    dict(dry=0.1 * (1 + k % 4), amp=0.1 + 0.1 * (k % 5), depth=2.0 + k % 6,
                         manning=0.02 + 0.005 * (k % 5),
                         scalars=2 if case["kind"] == "batch" else 1 + k % 3)))
    return out


def _build(deck, geometry="fine", precision="fp64"):
    cfg = deck["cfg"]
    dom = native.Domain(cfg)
    zf = deck["zf"].cpu().numpy()
    if geometry == "fine":
        dom.set_fine_bottoms(zf, R)
    else:
        ne = int(round((cfg["surfmax"] - cfg["surfmin"]) / cfg["dsurf"]))
        dom.set_tables(native.build_tables(zf, cfg["nx"], cfg["ny"], R, cfg["dxf"], cfg["dyf"],
                                           cfg["surfmin"], cfg["dsurf"], ne))
    dom.set_tide(deck["tide"])
    for kind, values in deck.get("series", {}).items():
        dom.set_series(kind, values)
    if precision == "mixed":
        dom.set_precision(native.PRECISION_MIXED, 1e-5)
    host = [deck[k].cpu().numpy().ravel() for k in ("bottom", "bxp", "byp", "surf")]
    dom.init(*host, None, None, deck["S"][0].cpu().numpy().ravel())
    for s in range(1, len(deck["S"])):
        dom.init_scalar(s, deck["S"][s].cpu().numpy().ravel())
    return dom


def _system(case, seed):
    """A free-surface system as a step assembles it: diagonal, east and north
    couplings, right-hand side; tidal and closed dry rows decoupled."""
    nx, ny = case["nx"], case["ny"]
    d = _deck(nx, ny, seed, dry=0.2)
    depth = (d["surf"] - d["bottom"]).clamp(min=0.0)
    hx, hy = torch.zeros_like(depth), torch.zeros_like(depth)
    hx[:, :-1] = (torch.maximum(d["surf"][:, :-1], d["surf"][:, 1:]) - d["bxp"][:, :-1]).clamp(min=0.0)
    hy[:-1] = (torch.maximum(d["surf"][:-1], d["surf"][1:]) - d["byp"][:-1]).clamp(min=0.0)
    Gx, Gy = G * hx, G * hy  # g dt^2 N^2 / V of a face with dt = 1
    Ct = 100.0 * torch.ones_like(depth) + Gx + Gy
    Ct[:, 1:] += Gx[:, :-1]
    Ct[1:] += Gy[:-1]
    noise = torch.randn(ny, nx, generator=_rng(seed, 3), dtype=torch.float64, device="cuda")
    b = 100.0 * (d["cfg"]["offset"] + d["surf"]) + noise
    off = (depth == 0) & (Ct == 100.0)
    off[-1] = True
    b[-1] = d["cfg"]["offset"]
    Ct[-1] = 1.0
    return [t.contiguous().view(-1) for t in (torch.where(off, -Ct, Ct), Gx, Gy, b)]


def prepare(case, seed):
    if case["kind"] == "solve":
        return {"case": case, "sys": _system(case, seed),
                "x": torch.zeros(case["nx"] * case["ny"], dtype=torch.float64, device="cuda")}
    if case["kind"] == "domain":
        return {"case": case, "t": 1,
                "dom": _build(_case_deck(case, seed), case["geometry"], case["precision"])}
    ms = _members(case, seed)
    doms = [_build(_deck(nx, ny, s, **kw), precision=case["precision"]) for nx, ny, _, s, kw in ms]
    host = (native.Batch if case["kind"] == "batch" else native.Server)(BUDGET, case["cells_per_cta"])
    return {"case": case, "host": host, "doms": doms, "t": [1] * len(doms), "steps": [m[2] for m in ms]}


# ------------------------------------------------------------------ one pass
def _fields(dom):
    out = dom.download(FIELDS)
    for s in range(1, dom.cfg["nscalar"]):
        out["S%d" % s] = dom.download_scalar(s)
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        ptrs = [t.data_ptr() for t in state["sys"]] + [state["x"].data_ptr()]
        native.cg_solve_noalloc(case["nx"], case["ny"], *ptrs, 1e-12, 100000)
        return state["x"]
    if case["kind"] == "domain":
        dom, t, n = state["dom"], state["t"], case["steps"]
        state["t"] = t + n
        if not case["stepwise"]:
            if dom.run(t, n) != 0:
                raise RuntimeError("the run stopped")
            return _fields(dom)
        seen = []
        for tt in range(t, t + n):
            if dom.step(tt) != 0:
                raise RuntimeError("the run stopped")
            st = dom.stats()
            seen += [st["volume"], st["max_cflx"], st["max_cfly"]]
        return dict(_fields(dom), seen=np.array(seen))
    if case["kind"] == "batch":
        b = state["host"]
        slots = [b.admit(d, t) for d, t in zip(state["doms"], state["t"])]
        for _ in range(case["steps"]):
            b.step()
        b.sync()
        for s in slots:
            b.release(s)
    else:
        srv = state["host"]
        for d, t, n in zip(state["doms"], state["t"], state["steps"]):
            srv.submit(d, n, t)
        done = 0
        while done < len(state["doms"]):
            for r in srv.poll(timeout_ms=1000):
                done += 1
                if r["status"] != 0:
                    raise RuntimeError("a request failed with status %d" % r["status"])
    state["t"] = [t + n for t, n in zip(state["t"], state["steps"])]
    # one vector per field over all basins
    parts = [_fields(d) for d in state["doms"]]
    names = sorted(set().union(*parts))
    return {k: np.concatenate([p[k] for p in parts if k in p]) for k in names}


# ------------------------------------------------------------------ compulsory work
def _step_work(cells, iters, mixed, scalars):
    """Bytes and operations one step of `cells` cells cannot do without: each
    stencil phase and each solver sweep reads its inputs and writes its outputs
    once (explicit phase 200 B, update phases 208 B, 16 B per further scalar;
    the solve 48 B, and 72 B per FP64 or 32 B per FP32 iteration)."""
    b = 408 + 16 * (scalars - 1) + 48 + (32 if mixed else 72) * iters
    return cells * b, cells * (600 + 40 * iters)


def work(case):
    if case["kind"] == "solve":
        # the system is read and x written once; on chip the iterations cost operations only
        n = case["nx"] * case["ny"]
        return {"bytes": 40.0 * n, "flops": 20.0 * 30 * n}
    if case["kind"] == "domain":
        n = case["nx"] * case["ny"]
        iters = 65 if case["dx"] < 5 else 30
        b, f = _step_work(n, iters, case["precision"] == "mixed", case["scalars"])
        return {"bytes": float(b * case["steps"] + 8 * n * (3 + case["scalars"])),
                "flops": float(f * case["steps"])}
    total = [0.0, 0.0]
    for nx, ny, steps, _, kw in _members(case, 0):
        b, f = _step_work(nx * ny, 30, case["precision"] == "mixed", kw["scalars"])
        total[0] += b * steps + 8.0 * nx * ny * (3 + kw["scalars"])
        total[1] += f * steps
    return {"bytes": total[0], "flops": total[1]}


# ------------------------------------------------------------------ 64-bit values
# The same results from plain torch in FP64: the scheme written array by array
# over the whole grid (ghost ring in place, cell (i, j) at [j + 1, i + 1]), with a
# textbook Jacobi-preconditioned CG.

def _sh(a, di=0, dj=0):
    ny, nx = a.shape[0] - 2, a.shape[1] - 2
    return a[1 + dj:1 + dj + ny, 1 + di:1 + di + nx]


def _pcg(Ct, Gx, Gy, b, eps, eliminate, x0=None):
    """Jacobi-PCG from x = 0 on the interior; Ct < 0 marks a decoupled row."""
    dec, D = Ct < 0, Ct.abs()
    keep = (~dec).double()

    def off(v):
        s = torch.zeros_like(v)
        s[:, :-1] += Gx[:, :-1] * v[:, 1:]
        s[:, 1:] += Gx[:, :-1] * v[:, :-1]
        s[:-1] += Gy[:-1] * v[1:]
        s[1:] += Gy[:-1] * v[:-1]
        return keep * s

    x = torch.zeros_like(b)
    r = b.clone()
    if eliminate:
        r = b + off(torch.where(dec, b / D, x))
    bn, p, rho, it = float(b.norm()), torch.zeros_like(b), 1.0, 0
    while float(r.norm()) >= eps * bn and it < 2000:
        z = r / D
        rho_new = float((r * z).sum())
        p = z + (rho_new / rho if it else 0.0) * p
        rho = rho_new
        q = D * p - off(keep * p if eliminate else p)
        a = rho / float((p * q).sum())
        x += a * p
        r -= a * q
        it += 1
    return x


class _Exact:
    """One domain's state and step."""

    def __init__(self, deck):
        c = self.c = deck["cfg"]
        self.zf, self.tide = deck["zf"], deck["tide"]
        ny, nx, off = c["ny"], c["nx"], c["offset"]
        self.ne = int(round((c["surfmax"] - c["surfmin"]) / c["dsurf"]))
        self.z0 = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
        self.z2 = torch.zeros(ny + 2, nx + 2, dtype=torch.float64, device="cuda")
        pad = self._pad
        self.bz, self.bx, self.by = (pad(deck[k] + off) for k in ("bottom", "bxp", "byp"))
        s = torch.maximum(deck["surf"] + off, _sh(self.bz))
        self.surf = pad(s)
        self._corners(self.surf)
        row = _sh(self.surf)[-1]
        h = float(self.tide[0]) + off
        row.copy_(torch.where(h > _sh(self.bz)[-1], torch.full_like(row, h), row))
        self.depth = pad((_sh(self.surf) - _sh(self.bz)).clamp(min=0.0))
        self.u, self.v = self.z2.clone(), self.z2.clone()
        self.cfx, self.cfy = self.z0.clone(), self.z0.clone()
        dep = _sh(self.depth)
        hx, hy = self._face_depths()
        co = G * c["manningN"] ** 2
        thin = co / dep.clamp(min=1e-300) ** (2.0 / 3.0)
        cd = torch.full_like(dep, c["CDx"])
        self.cdx = torch.where((dep > 0) & (hx <= c["hD"]), thin, cd)
        self.cdy = torch.where((dep > 0) & (hy <= c["hD"]), thin, cd)
        self.S = []
        for f in deck["S"]:
            a = self.z2.clone()
            _sh(a).copy_(torch.where(dep > 0, f, torch.zeros_like(f)))
            self.S.append(a)
        self.ind = torch.full((ny, nx), self.ne // 2, device="cuda")
        self._geometry(dep)
        self.surf = (self.surf - off) + off

    def _pad(self, a):
        b = self.z2.clone()
        _sh(b).copy_(a)
        b[0, 1:-1], b[-1, 1:-1] = a[0], a[-1]
        b[1:-1, 0], b[1:-1, -1] = a[:, 0], a[:, -1]
        return b

    @staticmethod
    def _corners(a):
        """The surface's corner ghosts, as the model fills them."""
        a[-1, -1], a[0, -1], a[-1, 0], a[0, 0] = a[-2, -1], a[-2, 0], a[1, -1], a[1, 0]

    def _face_depths(self):
        s = self.surf
        hx = (torch.maximum(_sh(s), _sh(s, 1)) - _sh(self.bx)).clamp(min=0.0)
        hy = (torch.maximum(_sh(s), _sh(s, 0, 1)) - _sh(self.by)).clamp(min=0.0)
        hx[:, -1] = 0.0
        hy[-1] = 0.0
        return hx, hy

    # -------------------------------------------------- subgrid geometry
    def _level_values(self, lev):
        """The ten table values of every cell at its level index."""
        c, ny, nx = self.c, self.c["ny"], self.c["nx"]
        h = c["surfmin"] + lev.double() * c["dsurf"]
        d = (h[:, None, :, None] - self.zf.view(ny, R, nx, R)).clamp_(min=0.0)
        dA, half = c["dxf"] * c["dyf"], R // 2
        zf = self.zf.view(ny, R, nx, R)
        o = {"V": dA * d.sum((1, 3)), "Z": dA * (d > 0).sum((1, 3)).double(),
             "Vxm": dA * d[..., :half].sum((1, 3)), "Vxp": dA * d[..., half:].sum((1, 3)),
             "Vym": dA * d[:, :half].sum((1, 3)), "Vyp": dA * d[:, half:].sum((1, 3))}

        def face(own, other, lv):  # other: the neighbour's pixels at this cell's level
            return torch.minimum(own, (lv - other).clamp(min=0.0))
        e, w = d[..., R - 1].clone(), d[..., 0].clone()      # (ny, R, nx)
        e[:, :, :-1] = face(e[:, :, :-1], zf[:, :, 1:, 0], h[:, None, :-1])
        w[:, :, 1:] = face(w[:, :, 1:], zf[:, :, :-1, R - 1], h[:, None, 1:])
        n, s = d[:, R - 1].clone(), d[:, 0].clone()          # (ny, nx, R)
        n[:-1] = face(n[:-1], zf[1:, 0], h[:-1, :, None])
        s[1:] = face(s[1:], zf[:-1, R - 1], h[1:, :, None])
        o["Np"], o["Nm"] = e.sum(1) * c["dxf"], w.sum(1) * c["dxf"]
        o["Op"], o["Om"] = n.sum(2) * c["dxf"], s.sum(2) * c["dxf"]
        return o

    def _geometry(self, depth_old):
        c, ne = self.c, self.ne
        s, ds = _sh(self.surf), c["dsurf"]
        levels = c["surfmin"] + torch.arange(ne, dtype=torch.float64, device="cuda") * ds + c["offset"]
        ind = self.ind
        for _ in range(ne + 2):
            lv = levels[ind]
            move = (lv - s).abs() > 0.5 * ds + ds / 100
            new = torch.where(move, torch.where(s > lv, ind + 1, ind - 1), ind).clamp(0, ne - 1)
            if torch.equal(new, ind):
                break
            ind = new
        self.ind = ind
        j2 = torch.where(s > levels[ind], ind + 1, ind - 1)
        j2 = torch.where((ind == 0) | (ind == ne - 1), ind, j2)
        a1, a2 = levels[ind], levels[j2]
        L1, L2 = self._level_values(ind), self._level_values(j2)
        same = j2 == ind

        def lin(x1, y1, y2):
            return torch.where(a2 == x1, y1, (y2 - y1) * (s - a2) / torch.where(a2 == x1, 1.0, a2 - x1) + y2)
        q = {k: lin(a1, L1[k], L2[k]) for k in ("V", "Z", "Vxp", "Vxm", "Vyp", "Vym")}
        edge = {"Np": _sh(self.bx).clone(), "Nm": _sh(self.bx, -1).clone(),
                "Op": _sh(self.by).clone(), "Om": _sh(self.by, 0, -1).clone()}
        edge["Nm"][:, 0] = 0.0
        edge["Om"][0] = 0.0
        for k, b in edge.items():
            inside = (b > a1) & (b < a2) & ~same
            f = torch.where(inside, torch.where(b > s, 0.0, lin(b, torch.zeros_like(b), L2[k])),
                            lin(a1, L1[k], L2[k]))
            shut = s - b <= 0
            if k == "Nm":
                shut[:, 0] = False
            if k == "Om":
                shut[0] = False
            q[k] = torch.where(shut, 0.0, f)
        for k in ("Vxp", "Vxm", "Vyp", "Vym"):
            q[k] = torch.where(depth_old == 0, 0.0, q[k])
        dxdy, Z = c["dx"] * c["dy"], q["Z"]

        def combine(p, m, va, vb, b, nxt):  # one direction, along dim `nxt`
            N, V, Zf = q[p].clone(), 2.0 * q[va], 2.0 * Z
            lo, hi = [slice(None)] * 2, [slice(None)] * 2
            lo[nxt], hi[nxt] = slice(None, -1), slice(1, None)
            lo, hi = tuple(lo), tuple(hi)
            N[lo] = torch.maximum(N[lo], q[m][hi])
            a, d = q[va][lo], q[vb][hi]
            v = torch.where((a > 0) & (d > 0), a + d, 2.0 * (a + d))
            z = Z[lo]
            z = torch.where((v > 0) & (z <= 0), dxdy, z)
            for cond, val in ((s[lo] < b[lo], d), (s[hi] < b[lo], a)):
                v = torch.where(cond, val, v)
                z = torch.where(cond, 0.5 * Z[lo], z)
            V[lo], Zf[lo] = v, z
            return N, V, Zf
        Nx, Vx, Zx = combine("Np", "Nm", "Vxp", "Vxm", _sh(self.bx), 1)
        Oy, Vy, Zy = combine("Op", "Om", "Vyp", "Vym", _sh(self.by), 0)

        def cut(a, to=0.0):
            return torch.where(a < 0.002, to, a)
        Nx, Oy, Vx, Vy, Zx, Zy = (self._pad(cut(a)) for a in (Nx, Oy, Vx, Vy, Zx, Zy))
        self.V, self.Z = cut(q["V"]), cut(Z, 1.0)
        Nx[:, 0] = Nx[:, -1] = 0.0
        Nx[1:-1, -2] = 0.0
        Oy[0] = 0.0  # the north row is tidal everywhere: its faces stay open
        self.Nx, self.Oy, self.Vx, self.Vy, self.Zx, self.Zy = Nx, Oy, Vx, Vy, Zx, Zy

    # -------------------------------------------------- one step
    def _interp(self):
        """velocityInterp with the reference's linear-index neighbours."""
        u, v = self.u, self.v
        b, d = _sh(u, -1).clone(), _sh(u, -1, 1).clone()
        b[1:, 0], b[0, 0] = _sh(u)[:-1, -1], 0.0
        d[:, 0] = _sh(u)[:, -1]
        uy = 0.25 * (_sh(u) + b + _sh(u, 0, 1) + d)
        b, a, d = _sh(v, 1).clone(), _sh(v, 0, -1).clone(), _sh(v, 1, -1).clone()
        b[:, -1] = _sh(v, 0, 1)[:, 0]
        a[0], d[0] = 0.0, 0.0
        d[:, -1] = _sh(v)[:, 0]
        vx = 0.25 * (_sh(v) + b + a + d)
        return uy, vx

    def _explicit(self, w, x_dir, uu, vv, cf, V, Z, cd):
        """Explicit momentum of one component: advection with the CFL limiter,
        diffusion, drag.  w: the component; uu, vv: advecting velocities."""
        c = self.c
        w0, E, W, N, S = _sh(w), _sh(w, 1), _sh(w, -1), _sh(w, 0, 1), _sh(w, 0, -1)
        ax = (0.5 / c["dx"]) * ((uu + uu.abs()) * (w0 - W) + (uu - uu.abs()) * (E - w0)) \
            + (0.5 / c["dy"]) * ((vv + vv.abs()) * (w0 - S) + (vv - vv.abs()) * (N - w0))
        ax = torch.where(w0 == 0, 0.0, ax)
        lo, hi = c["CFLl"], c["CFLh"]
        for di, dj in ((0, 1), (1, 0), (0, 0)):  # the row before, the column before, the cell
            f, fx = torch.zeros_like(cf), torch.zeros_like(cf)
            f[dj:, di:], fx[dj:, di:] = cf[:cf.shape[0] - dj, :cf.shape[1] - di], \
                self.cfx[:cf.shape[0] - dj, :cf.shape[1] - di]
            soft = (f > lo) & ((f <= hi) if x_dir else (f < hi))
            cutoff = (f > hi) if x_dir else (fx > hi)
            ax = torch.where(soft, ax * (hi - cf) / (hi - lo), torch.where(cutoff, 0.0, ax))
        En = w0 - c["dt"] * ax
        V0 = _sh(V)
        Vs = torch.where(V0 > 0, V0, 1.0)
        if x_dir:
            fl = (c["NUx"] / Vs) * (_sh(self.Nx, 1) * (E - w0) - _sh(self.Nx) * (w0 - W)) / c["dx"] + \
                (c["NUy"] / Vs) * (_sh(self.Oy) * (N - w0) - _sh(self.Oy, 0, -1) * (w0 - S)) / c["dy"]
        else:
            fl = (c["NUx"] / Vs) * (_sh(self.Nx) * (E - w0) - _sh(self.Nx, -1) * (w0 - W)) / c["dx"] + \
                (c["NUy"] / Vs) * (_sh(self.Oy, 0, 1) * (N - w0) - _sh(self.Oy) * (w0 - S)) / c["dy"]
        En = En + c["dt"] * torch.where(V0 > 0, fl, 0.0)
        drag = 0.5 * c["dt"] * cd * (uu * uu + vv * vv).sqrt() * torch.where(V0 > 0, _sh(Z) / Vs, 0.0)
        return En / (1 + drag), drag

    def step(self, tt):
        c = self.c
        g, dt, dx, dy, off = G, c["dt"], c["dx"], c["dy"], c["offset"]
        tide = float(self.tide[tt]) + off
        uy, vx = self._interp()
        Enx, Dx = self._explicit(self.u, True, _sh(self.u), vx, self.cfx, self.Vx, self.Zx, self.cdx)
        Eny, Dy = self._explicit(self.v, False, uy, _sh(self.v), self.cfy, self.Vy, self.Zy, self.cdy)

        # ---- assembly
        def coupling(N, V, D):
            return torch.where(_sh(V) > 0, g * dt * dt * _sh(N) ** 2 /
                               torch.where(_sh(V) > 0, _sh(V), 1.0) / (1 + D), 0.0)
        Gx, Gy = coupling(self.Nx, self.Vx, Dx), coupling(self.Oy, self.Vy, Dy)
        Gw, Gs = torch.zeros_like(Gx), torch.zeros_like(Gy)
        Gw[:, 1:], Gs[1:] = Gx[:, :-1], Gy[:-1]
        s = _sh(self.surf)
        Fx, Fy = Enx * _sh(self.Nx), Eny * _sh(self.Oy)
        div = Fx + Fy
        div[:, 1:] -= Fx[:, :-1]
        div[1:] -= Fy[:-1]
        b = s * self.Z - dt * div
        b = torch.where(b == 0, s * dx * dy, b)
        Ct = self.Z + Gx + Gy + Gw + Gs
        Ct = torch.where(Ct == 0, dx * dy, Ct)
        shut = (_sh(self.depth) == 0) & (_sh(self.u) == 0) & (_sh(self.u, -1) == 0) & \
            (_sh(self.v) == 0) & (_sh(self.v, 0, -1) == 0)
        Ct = torch.where(shut, dx * dy, Ct)
        b = torch.where(shut, s * dx * dy, b)
        Ct[:, -1] -= torch.where(shut[:, -1], 0.0, Gx[:, -1])
        shut[-1] = True
        Ct[-1], b[-1] = 1.0, tide
        Gx[:, -1], Gy[-1] = 0.0, 0.0
        x = _pcg(torch.where(shut, -Ct, Ct), Gx, Gy, b, c["eps"], False)

        # ---- surface
        bz = _sh(self.bz)
        pre = torch.maximum(x, bz)
        ns = pre.clone()
        ns[-1] = torch.where(tide > bz[-1], torch.full_like(ns[-1], tide), ns[-1])
        so = s + c["minDepth"]
        alone = (_sh(self.depth) <= 0) & (ns - bz > 0)
        dep0 = self.z2.clone()  # depth's ghosts are never written
        _sh(dep0).copy_(_sh(self.depth))
        for di, dj in ((1, 0), (-1, 0), (0, 1), (0, -1)):
            alone &= (_sh(self.surf, di, dj) <= so) | (_sh(dep0, di, dj) <= 0)
        ns = torch.where(alone, bz, ns)
        ns = torch.where((ns - bz <= c["minDepth"]) & (ns - bz > 0), bz, ns)
        old, depth_old, V_old = self.surf, _sh(self.depth), self.V
        new = self._pad(pre)
        _sh(new).copy_(ns)
        self._corners(new)
        self.surf = new
        self.depth = self._pad((ns - bz).clamp(min=0.0))
        self._geometry(depth_old)

        # ---- velocities
        def face(En, N, V, b, di, dj, w):
            N0, V0 = _sh(N), _sh(V)
            sn = _sh(self.surf, di, dj)
            f = En - g * dt * torch.where(V0 > 0, N0 / torch.where(V0 > 0, V0, 1.0), 0.0) * (sn - ns)
            f = torch.where(N0 == 0, 0.0, f)
            dep = _sh(self.depth)
            f = torch.where((dep == 0) & (f > 0), 0.0, f)
            inner = torch.ones_like(dep, dtype=torch.bool)
            if di:
                inner[:, -1] = False
            else:
                inner[-1] = False
            f = torch.where(inner & (_sh(self.depth, di, dj) == 0) & (f < 0), 0.0, f)
            rm = torch.zeros(alone.shape[0] + 2, alone.shape[1] + 2, dtype=torch.bool, device="cuda")
            _sh(rm).copy_(alone)
            f = torch.where(alone | (inner & _sh(rm, di, dj)), 0.0, f)
            b = _sh(b)
            fall = torch.where((ns < b) & (sn - b >= c["wtfh"]), -1.0, 0.0)
            fall = torch.where(inner & (sn < b) & (ns - b >= c["wtfh"]), 1.0, fall)
            top = 0.24 / c["subR"] * dx / dt
            wf = (0.7 * (2 * g * N0 / w).sqrt()).clamp(max=top)
            return torch.where(fall != 0, fall * wf, f)
        uE = face(Enx, self.Nx, self.Vx, self.bx, 1, 0, dy)
        vN = face(Eny, self.Oy, self.Vy, self.by, 0, 1, dx)
        uW, vS = uE.clone(), vN.clone()
        uW[:, 1:], vS[1:] = uE[:, :-1], vN[:-1]
        Nx, Oy, NxW, OyS = _sh(self.Nx), _sh(self.Oy), _sh(self.Nx, -1), _sh(self.Oy, 0, -1)
        FE, FW, FN, FS = uE * Nx, uW * NxW, vN * Oy, vS * OyS
        vst = vN.clone()
        rest = (FS + FW - FE - (ns - _sh(old)) * self.Z / dt)[-1]
        open_ = (rest != 0) & (Oy[-1] > 0)
        vst[-1] = torch.where(open_, rest / torch.where(open_, Oy[-1], 1.0), 0.0)
        self.u, self.v = self._pad(uE), self._pad(vN)
        _sh(self.v).copy_(vst)
        u, v = self.u, self.v
        u[-1, -1], u[0, -1], u[-1, 0], u[0, 0] = uE[-1, -1], uE[0, -1], uE[-1, 0], uE[0, 0]
        v[-1, -1], v[0, -1], v[-1, 0], v[0, 0] = vN[-1, -1], vN[-1, 0], vN[0, -1], vN[0, 0]
        cv = (V_old + dt * (FW - FE + FS - FN)).clamp(min=0.0)

        # ---- drag
        co = g * c["manningN"] ** 2
        wet = self.V > 0
        cd = co / torch.where(wet, self.V / self.Z, 1.0) ** (1.0 / 3.0)
        dep = _sh(self.depth)
        thin = co / torch.where(dep > 0, dep, 1.0) ** (2.0 / 3.0)
        hx, hy = self._face_depths()
        self.cdx = torch.where((dep > 0) & (hx <= c["hD"]), thin, torch.where(wet, cd, self.cdx))
        self.cdy = torch.where((dep > 0) & (hy <= c["hD"]), thin, torch.where(wet, cd, self.cdy))

        # ---- scalars
        h = old - self.bz
        north = torch.ones_like(dep, dtype=torch.bool)
        north[-1, 1:] = False
        south = torch.ones_like(north)
        south[0] = False
        near = [(1, 0, (Nx > 0) & (_sh(h, 1) > 0)), (-1, 0, (NxW > 0) & (_sh(h, -1) > 0)),
                (0, 1, north & (Oy > 0) & (_sh(h, 0, 1) > 0)), (0, -1, south & (OyS > 0) & (_sh(h, 0, -1) > 0))]
        dry = torch.zeros_like(north)
        for q, S in enumerate(self.S):
            Sc, SE, SW, SN, SS = _sh(S), _sh(S, 1), _sh(S, -1), _sh(S, 0, 1), _sh(S, 0, -1)
            m = Sc * V_old + dt * (-FE * torch.where(FE > 0, Sc, SE) + FW * torch.where(FW > 0, SW, Sc)
                                   - FN * torch.where(FN > 0, Sc, SN) + FS * torch.where(FS > 0, SS, Sc))
            m = m + dt * (c["Kx"] / dx * (Nx * (SE - Sc) - NxW * (Sc - SW)) +
                          c["Ky"] / dy * (Oy * (SN - Sc) - OyS * (Sc - SS)))
            Sn = torch.where(cv > 0, m / torch.where(cv > 0, cv, 1.0), 0.0)
            top, bot = torch.full_like(Sn, -math.inf), torch.full_like(Sn, math.inf)
            for di, dj, ok in near:
                top = torch.where(ok, torch.maximum(top, _sh(S, di, dj)), top)
                bot = torch.where(ok, torch.minimum(bot, _sh(S, di, dj)), bot)
            some = near[0][2] | near[1][2] | near[2][2] | near[3][2]
            Sn = torch.where(some, torch.minimum(torch.maximum(Sn, bot), top), Sn)
            odd = (Sn > 100) | (Sn < 0)
            odd[0] = False
            odd[-1, 1:] = False
            Sn = torch.where(odd, 0.0, Sn)
            if q == 0:
                dry = odd
            T = self._pad(Sn)
            T[0, 0], T[0, -1], T[-1, 0], T[-1, -1] = S[0, 0], S[0, -1], S[-1, 0], S[-1, -1]
            Sn = Sn.clone()
            Sn[-1] = c["tidePS"]
            _sh(T).copy_(torch.where((dep <= 0) | (odd if q == 0 else False), 0.0, Sn))
            self.S[q] = T
        _sh(self.surf).copy_(torch.where(dry, ns - dep, ns))
        _sh(self.depth).copy_(torch.where(dry, 0.0, dep))
        self.cfx, self.cfy = uE.abs() * dt / dx, vst.abs() * dt / dy
        return [float(cv.sum()), float(self.cfx.max()), float(self.cfy.max())]

    def fields(self):
        """The state in the order the framework hands it out: interior, then the
        north, south, east and west ghosts and the corners."""
        out = {"surf": self.surf, "uuXP": self.u, "vvYP": self.v, "S": self.S[0]}
        out.update({"S%d" % s: a for s, a in enumerate(self.S) if s})
        return {k: torch.cat([_sh(a).flatten(), a[-1, 1:-1], a[0, 1:-1], a[1:-1, -1], a[1:-1, 0],
                              torch.stack([a[-1, 0], a[-1, -1], a[0, -1], a[0, 0]])]).cpu().numpy()
                for k, a in out.items()}


def exact(case, seed):
    if case["kind"] == "solve":
        ny, nx = case["ny"], case["nx"]
        Ct, Gx, Gy, b = (t.view(ny, nx) for t in _system(case, seed))
        return _pcg(Ct, Gx, Gy, b, 1e-15, True).view(-1)
    if case["kind"] == "domain":
        if case["forced"] or case["adv"] != 1:
            return None  # the options are not restated here
        e, seen = _Exact(_case_deck(case, seed)), []
        for tt in range(1, case["steps"] + 1):
            seen += e.step(tt)
        out = e.fields()
        return dict(out, seen=np.array(seen)) if case["stepwise"] else out
    if sum(nx * ny for nx, ny, *_ in _members(case, seed)) * case["steps"] > 80e6:
        return None  # over the time it may take
    parts = []
    for nx, ny, steps, s, kw in _members(case, seed):
        e = _Exact(_deck(nx, ny, s, **kw))
        for tt in range(1, steps + 1):
            e.step(tt)
        parts.append(e.fields())
    names = sorted(set().union(*parts))
    return {k: np.concatenate([p[k] for p in parts if k in p]) for k in names}

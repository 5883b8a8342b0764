"""The work whose time counts here: what users of this framework have it do, through the calls of
``amber_b200``, over the sizes of its configurations (128² x 32 channels up to 512² x 384 channels, the
ensemble's sides 96-320 with 24-160 channels, the serving stream's sides 64-384 with 16-256 channels).

A case is a dict of plain values; its ``kind`` names the call:

* ``triangle``     file-ready sums of one triangle (``Estimator.triangle_v1`` / ``triangle_v2``): the body of the
                   drop-in executable's loop;
* ``triangles``    FP64 lag arrays of a run of triangles (``Estimator.triangles``), mixed or plain FP64;
* ``realisation``  one realisation from host arrays to lag arrays: grid, rings, channels, calCR, every triangle;
* ``ensemble``     realisations of uneven size through the request engine, cubes resident on the device;
* ``grid``         visibility records from host memory onto the grid, with or without channel collapse;
* ``maps``         the MAPS two-point function of the loaded grid;
* ``cylbs``        cylindrical bispectra of a finished run.

Inputs follow the synthetic recipe of ``amber_b200.synth`` (power law in |U|, channels correlated over
eight channels, Poisson sampling counts, flagged channels without samples, a Hermitian j = 0 column), drawn
on the device so that they are quick to make.
"""
import math

import numpy as np
import torch

import amber_b200
from amber_b200 import Engine, Estimator
from amber_b200.synth import NU0, Realisation

DU = 0.5
# the declared ranges keep a drawn case's lag-triple products below these, by kind
MOST_PRODUCTS = {"mixed": 7.0e12, "fp64": 3.0e11, "ensemble": 9.0e12, "cylbs": 3.0e11}


# ---- geometry: rings, closed triangles, map sides, flags ------------------------------------------------------

def edges(case):
    e = np.geomspace(2.0, case["ring_hi"], case["nbins"] + 1)
    e[0], e[-1] = 2.0, case["ring_hi"]
    return e[:-1].copy(), e[1:].copy()


def closed(case):
    lo, hi = edges(case)
    ua = [(2.0 / 3.0) * (math.pow(b, 3.0) - math.pow(a, 3.0)) / (math.pow(b, 2.0) - math.pow(a, 2.0))
          for a, b in zip(lo.tolist(), hi.tolist())]
    out = []
    for r1 in range(len(ua)):
        for r2 in range(r1 + 1):
            t = ua[r2] / ua[r1]
            if not 0.5 <= t <= 1.0:
                continue
            for r3 in range(r2 + 1):
                mu = 0.5 * (t + 1.0 / t - (ua[r3] / ua[r1]) * (ua[r3] / ua[r2]))
                if 0.5 / t <= mu <= 1.0:
                    out.append((r1, r2, r3))
    return out


def side_of(hi):
    n = int(3 * int((hi + 3) / DU))
    return n + 2 if n % 2 == 0 else n + 3


def flags(case):
    """Flagged channels: ``flagged`` of them, at places that depend on the channel count alone."""
    nc = case["nc"]
    if not case["flagged"]:
        return None
    rng = np.random.default_rng(7919 + nc)
    return np.sort(rng.choice(nc, size=max(1, int(round(case["flagged"] * nc))), replace=False))


def weights(case):
    w = np.ones(case["nc"])
    f = flags(case)
    if f is not None:
        w[f] = 0.0
    return w


def triplets(case):
    """Channel triplets of one triangle: sum over anchors of (window population)^2."""
    w, n = weights(case), case["nc10"]
    c = np.concatenate([[0.0], np.cumsum(w)])
    p = np.arange(case["nc"])
    inside = c[np.minimum(case["nc"], p + n + 1)] - c[np.maximum(0, p - n)]
    return float((w * inside * inside).sum())


def chosen(case):
    tri = closed(case)
    if case.get("kind") == "cylbs":
        # rings wide enough that every mask sum the analysis divides by is made of many triads
        return [t for t in tri if t[2] >= 3]
    return tri[case["first"]:case["first"] + case["count"]] if "first" in case else tri


def products(case):
    """Lag-triple products of one pass over the case's triangles (and mask sums with version 2)."""
    _, hi = edges(case)
    return triplets(case) * sum(side_of(hi[t[0]]) ** 2 for t in chosen(case)) * case["version"]


# ---- the cases ------------------------------------------------------------------------------------------------

def sky(nn, nc, nbins, nc10=None, flagged=0.1, ring_hi=None):
    return {"nn": nn, "nc": nc, "nbins": nbins, "nc10": nc // 2 - 1 if nc10 is None else nc10, "flagged": flagged,
            "ring_hi": float(math.floor(0.47 * nn)) if ring_hi is None else ring_hi}


# four shapes of the 64-realisation ensemble, sides 96-192
MIX = ((96, 131), (128, 47), (96, 86), (192, 60))


def mix(case):
    return [sky(nn, nc, 12) | {"version": 2} for nn, nc in MIX[:case["requests"]]] if "sides" not in case else [
        sky(int(nn), int(nc), 12) | {"version": 2}
        for nn, nc in zip(case["sides"].split(","), case["channels"].split(","))]


def listed():
    return [
        # the smallest call: one triangle of the serving stream's smallest realisations, latency counts
        {"name": "one_small_triangle", "kind": "triangle", **sky(64, 16, 6), "first": 2, "count": 1, "version": 1},
        # the drop-in's per-triangle loop at the single realisation's size, with sampling-mask sums
        {"name": "one_triangle_v2", "kind": "triangle", **sky(256, 128, 16, flagged=0.125, ring_hi=120.0),
         "first": 150, "count": 1, "version": 2},
        # the reference's CPU-runnable configuration whole, widest lag window, every triangle
        {"name": "cpu_case_mixed", "kind": "triangles", "precision": "mixed",
         **sky(128, 32, 8, nc10=31, flagged=0.0, ring_hi=60.0), "version": 1},
        # the same on the plain FP64 path, which checks the mixed one
        {"name": "cpu_case_fp64", "kind": "triangles", "precision": "fp64",
         **sky(128, 32, 8, nc10=31, flagged=0.0, ring_hi=60.0), "version": 1},
        # the largest maps of the single realisation (Ng1 = 740)
        {"name": "widest_maps_v1", "kind": "triangles", "precision": "mixed",
         **sky(256, 128, 16, flagged=0.125, ring_hi=120.0), "first": 196, "count": 20, "version": 1},
        # the large cube's channel count: lag windows of three tiles a side
        {"name": "wide_window_v2", "kind": "triangles", "precision": "mixed",
         **sky(256, 384, 12, flagged=0.15, ring_hi=60.0), "first": 60, "count": 10, "version": 2},
        # plain FP64 at the single realisation's channel count
        {"name": "fp64_triangles_v2", "kind": "triangles", "precision": "fp64",
         **sky(256, 128, 16, flagged=0.125, ring_hi=120.0), "first": 90, "count": 6, "version": 2},
        # one realisation of the ensemble from host arrays to results
        {"name": "realisation_v2", "kind": "realisation", **sky(128, 59, 12), "version": 2},
        # a batch of the ensemble through the request engine
        {"name": "ensemble_v2", "kind": "ensemble", "requests": 4},
        # the gridding stage: records from host memory onto the 256² grid
        {"name": "gridding", "kind": "grid", "nn": 256, "nc": 128, "records": 40000, "flag_key": 1, "collapse": 1},
        # MAPS two-point function at the single realisation's size
        {"name": "maps_two_point", "kind": "maps", **sky(256, 128, 16, flagged=0.125, ring_hi=120.0), "bins": 15},
        # cylindrical bispectra of a v2 run, windowed, as the analysis stage makes them
        {"name": "cylindrical", "kind": "cylbs", **sky(128, 112, 8, ring_hi=20.0), "n_cut": 8, "version": 2},
    ]


def spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["triangle", "triangles", "triangles", "triangles", "triangles", "realisation", "ensemble",
                       "grid", "maps", "cylbs"])
    nn = 2 * spread(rng, 32, 160)
    nc = spread(rng, 16, 256)
    if kind == "grid":
        return {"kind": kind, "nn": nn, "nc": min(nc, 128), "records": spread(rng, 200, 40000),
                "flag_key": rng.randint(0, 1), "collapse": rng.choice([1, 1, 4])}
    if kind == "maps":
        return {"kind": kind, **sky(min(nn, 256), min(nc, 128), 8), "bins": rng.randint(5, 20)}
    if kind == "ensemble":
        sides = [2 * spread(rng, 32, 96) for _ in range(rng.randint(2, 4))]
        chans = [spread(rng, 24, 160) for _ in sides]
        case = {"kind": kind}
        while True:
            case |= {"sides": ",".join(map(str, sides)), "channels": ",".join(map(str, chans))}
            if sum(products(c) for c in mix(case)) <= MOST_PRODUCTS[kind]:
                return case
            chans = [max(24, 3 * c // 4) for c in chans]
            sides = [max(64, 2 * (2 * s // 5)) for s in sides]
    case = {"kind": kind, **sky(nn, nc, rng.randint(6, 16), flagged=rng.choice([0.0, 0.1, 0.15])),
            "version": rng.randint(1, 2)}
    if rng.random() < 0.15:
        case["nc10"] = min(case["nc"] - 1, 95)  # the widest lag window the channel count allows
    if kind == "realisation":
        case |= sky(min(nn, 128), min(nc, 64), 8) | {"kind": kind}
        return case
    if kind == "cylbs":
        while True:
            case |= sky(min(nn, 128), max(24, min(nc, 128)), 8, ring_hi=min(20.0, float(math.floor(0.47 * nn))))
            case["n_cut"] = rng.choice([1, 2, 8]) if case["nc10"] > 11 else 1
            if products(case) <= MOST_PRODUCTS[kind]:
                return case
            nc = 3 * min(nc, 128) // 4
    if kind == "triangles":
        case["precision"] = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    most = MOST_PRODUCTS[case.get("precision", "mixed")]
    n = len(closed(case))
    case["first"] = rng.randrange(n)
    case["count"] = 1 if kind == "triangle" else rng.randint(1, 40)
    case["count"] = min(case["count"], n - case["first"])
    while products(case) > most and (case["count"] > 1 or case["first"] > 0):
        case["count"] = max(1, case["count"] // 2)
        case["first"] //= 2
    return case


# ---- inputs ---------------------------------------------------------------------------------------------------

def cube(case, seed):
    """Summed visibilities complex128 [NN, NN/2+1, nc] and counts float64, on the device."""
    nn, nc, h = case["nn"], case["nc"], case["nn"] // 2 + 1
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(1000003 * int(seed) + 31 * nn + nc)

    def normal(*shape):
        return torch.complex(torch.randn(*shape, generator=g, device=dev, dtype=torch.float64),
                             torch.randn(*shape, generator=g, device=dev, dtype=torch.float64)) / math.sqrt(2.0)

    ia = torch.arange(nn, device=dev, dtype=torch.float64)
    ia = torch.where(ia > nn // 2, ia - nn, ia)
    u = torch.sqrt(ia[:, None] ** 2 + torch.arange(h, device=dev, dtype=torch.float64)[None, :] ** 2)
    amp = torch.where(u > 0, u.clamp(min=0.5) ** -1.25, torch.zeros_like(u))
    rho = math.exp(-1.0 / 8.0)
    gv = torch.empty(nn, h, nc, dtype=torch.complex128, device=dev)
    x = normal(nn, h)
    for c in range(nc):
        if c:
            x = rho * x + math.sqrt(1.0 - rho * rho) * normal(nn, h)
        gv[:, :, c] = x * amp
    rms = float(gv.abs().square().mean().sqrt())
    lam = 4.0 * torch.exp(-u / (20.0 * nn / 128.0))
    lam[(u > case["ring_hi"]) | (u == 0)] = 0.0
    counts = torch.poisson(lam[:, :, None].expand(nn, h, nc).contiguous(), generator=g)
    gv = counts * gv + counts.sqrt() * (0.1 * rms) * normal(nn, h, nc)
    f = flags(case)
    if f is not None:
        f = torch.as_tensor(f, device=dev)
        counts[:, :, f] = 0.0
        gv[:, :, f] = 0.0
    k = torch.arange(1, nn // 2, device=dev)
    gv[nn - k, 0] = gv[k, 0].conj()
    counts[nn - k, 0] = counts[k, 0]
    gv[0, 0] = 0.0
    counts[0, 0] = 0.0
    gv[nn // 2, 0] = gv[nn // 2, 0].real.to(gv.dtype)
    return gv.contiguous(), counts.contiguous()


def channels(case):
    f = flags(case)
    return None if f is None else np.setdiff1d(np.arange(case["nc"]), f).astype(np.int32)


def ready(case, seed, precision="mixed"):
    """An Estimator with the case's grid, rings and channels."""
    gv, counts = cube(case, seed)
    est = Estimator(precision=precision)
    torch.cuda.synchronize()
    est.load_grid_device(gv.data_ptr(), counts.data_ptr(), case["nn"], case["nc"], DU, int(channels(case) is not None))
    est.set_rings(*edges(case))
    est.set_channels(case["nc10"], channels(case))
    return est


def host(case, seed, with_cube=True):
    gv, counts = cube(case, seed)
    lo, hi = edges(case)
    uf = channels(case)
    real = Realisation(nn=case["nn"], nc=case["nc"], du=DU, flag_key=int(uf is not None),
                       gv=gv.cpu().numpy() if with_cube else np.broadcast_to(np.zeros(1, np.complex128), gv.shape),
                       counts=counts.cpu().numpy() if with_cube else np.broadcast_to(np.zeros(1), counts.shape),
                       uf_chans=np.arange(case["nc"], dtype=np.int32) if uf is None else uf, ulow=lo, uhigh=hi,
                       nc10=case["nc10"], seed=seed)
    return real, gv, counts


def records(case, seed):
    """randpar float32 [G, 3] and data float32 [G, nc, 2, 3]; a third of the records fall on an earlier one's cell."""
    nn, g = case["nn"], case["records"]
    rng = np.random.default_rng(int(seed))
    umax = 0.95 * DU * (nn // 2)
    r, th = umax * np.sqrt(rng.uniform(0, 1, g)), rng.uniform(-math.pi, math.pi, g)
    u, v = r * np.cos(th), r * np.sin(th)
    src, dst = rng.integers(0, g, g // 3), rng.integers(0, g, g // 3)
    u[dst], v[dst] = u[src], v[src]
    randpar = np.zeros((g, 3), dtype=np.float32)
    randpar[:, 0], randpar[:, 1] = u / NU0, v / NU0
    data = rng.standard_normal((g, case["nc"], 2, 3), dtype=np.float32)
    data *= np.float32(10.0)
    wt = data[..., 2]
    np.abs(wt, out=wt)
    wt[wt < 1.2566] = -1.0  # a tenth of the weights are flagged
    return randpar, data, umax


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        randpar, data, umax = records(case, seed)
        return {"kind": kind, "case": case, "est": Estimator(), "randpar": randpar, "data": data, "umax": umax}
    if kind == "ensemble":
        reqs = [host(c, 17 * seed + i, with_cube=False) for i, c in enumerate(mix(case))]
        est = Estimator(precision="mixed")
        torch.cuda.synchronize()
        return {"kind": kind, "est": est, "engine": Engine(est), "reqs": reqs}
    if kind == "realisation":
        real, _, _ = host(case, seed)
        return {"kind": kind, "est": Estimator(precision="mixed"), "real": real, "version": case["version"]}
    est = ready(case, seed, "fp64" if kind == "cylbs" else case.get("precision", "mixed"))
    state = {"kind": kind, "est": est, "case": case}
    if kind in ("triangle", "triangles", "cylbs"):
        state["tri"] = np.array(chosen(case), dtype=np.int32)
    if kind == "triangle":
        state["num"] = 1.0e6  # calCR's Num of the triangle, which the caller has read from its file
    if kind == "cylbs":
        est.run(state["tri"], want_v2=case["version"] == 2)
    return state


def run(state):
    kind, est = state["kind"], state["est"]
    if kind == "triangle":
        r1, r2, r3 = (int(r) for r in state["tri"][0])
        if state["case"]["version"] == 1:
            return est.triangle_v1(r1, r2, r3, state["num"])
        return est.triangle_v2(r1, r2, r3)
    if kind == "triangles":
        return est.triangles(state["tri"], want_v2=state["case"]["version"] == 2)
    if kind == "realisation":
        rdata, res = amber_b200.estimate(state["real"], version=state["version"], est=est)
        out = [rdata, np.stack([r["bldnu"] for r in res]), np.stack([r["numdnu"] for r in res])]
        return out + ([np.stack([r["numtri"] for r in res])] if state["version"] == 2 else [])
    if kind == "ensemble":
        eng = state["engine"]
        tickets = [eng.enqueue(real, True, device_cube=(gv.data_ptr(), counts.data_ptr()))
                   for real, gv, counts in state["reqs"]]
        return [eng.result(t, real, True)[:4] for t, (real, _, _) in zip(tickets, state["reqs"])]
    if kind == "grid":
        c = state["case"]
        return est.grid_vis(c["nn"], c["nc"], DU, state["umax"], NU0, c["flag_key"], state["randpar"], state["data"],
                            n_collapse=c["collapse"])
    if kind == "maps":
        return est.cl_dnu(state["case"]["bins"], 1.0, 0.5 * DU * state["case"]["nn"])
    c = state["case"]
    return est.cyl_bs(window=c["version"] == 2, denominator="mask" if c["version"] == 2 else "counts",
                      n_cut=c["n_cut"])


# ---- the least that a pass moves and computes -----------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        each = [work(c | {"kind": "realisation"}) for c in mix(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    nn, nc = case["nn"], case["nc"]
    cells = nn * (nn // 2 + 1)
    if kind == "grid":
        g = case["records"]
        return {"bytes": 8.0 * g + 12.0 * g * nc + 24.0 * cells * (nc // case["collapse"]), "flops": 3.0 * g * nc}
    if kind == "maps":
        u = np.hypot(np.minimum(np.arange(nn), nn - np.arange(nn))[:, None], np.arange(nn // 2 + 1)[None, :]) * DU
        inside = int(((u >= 1.0) & (u < 0.5 * DU * nn)).sum())
        return {"bytes": 24.0 * inside * nc + 8.0 * case["bins"] * nc, "flops": 5.0 * inside * nc * (nc + 1) / 2}
    tri, nclen = chosen(case), 2 * case["nc10"] + 1
    lags = 8.0 * nclen * nclen * len(tri) * case["version"]
    if kind == "cylbs":
        m, n = case["nc10"] + 1 - case["n_cut"], nclen - 2 * case["n_cut"]
        return {"bytes": lags + 8.0 * n * n * len(tri), "flops": 8.0 * m * n * n * len(tri)}
    _, hi = edges(case)
    ring = sum(2.0 * math.pi * hi[t[0]] ** 2 for t in {(t[0],) for t in tri})
    return {"bytes": float(min(24.0 * cells, 24.0 * ring) * nc + lags), "flops": 2.0 * products(case)}


# ---- the same in 64 bits, in plain torch and numpy ------------------------------------------------------------

def planes(grid, lo, hi, ng):
    """Maps [nc, ng, ng] of one ring: the ring's cells on an ng-point half plane, then an unnormalised c2r."""
    nn, h, nc = grid.shape
    dev = grid.device
    top = min(ng // 3, h)
    # membership on the host: a cell on an edge is decided by the correctly rounded square root
    ia, jj = np.arange(-(ng // 2) + 1, ng // 2 + 1), np.arange(top)
    u = np.sqrt((ia[:, None] ** 2 + jj[None, :] ** 2).astype(np.float64))
    i, j = np.nonzero((u >= lo) & (u < hi) & (u > 0))
    at, j = torch.as_tensor(ia[i], device=dev), torch.as_tensor(jj[j], device=dev)
    half = torch.zeros(nc, ng, ng // 2 + 1, dtype=torch.complex128, device=dev)
    half[:, at % ng, j] = grid[at % nn, j].T.to(torch.complex128)
    y = torch.fft.ifft(half, dim=1, norm="forward")
    y[:, :, 0] = y[:, :, 0].real.to(y.dtype)
    return torch.fft.irfft(y, n=ng, dim=2, norm="forward")


def lag_sums(case, grid, tri):
    """[ntri, nclen, nclen] sums of D1·D2·D3 over pixels and anchors, in the order of ``tri``."""
    nc, n, nclen = case["nc"], case["nc10"], 2 * case["nc10"] + 1
    lo, hi = edges(case)
    live = weights(case)
    w = torch.as_tensor(live, device=grid.device)
    out = torch.zeros(len(tri), nclen, nclen, dtype=torch.float64, device=grid.device)
    kept, ng_kept = {}, 0
    for t, (r1, r2, r3) in enumerate(tri):
        ng = side_of(hi[r1])
        if ng != ng_kept:
            kept, ng_kept = {}, ng
        need = {r: kept.get(r) for r in (r1, r2, r3)}
        if len(kept) * nc * ng * ng * 8 > 2e10:
            kept = {}
        for r in need:
            if need[r] is None:
                chunk = 4096
                m = planes(grid, lo[r], hi[r], ng).reshape(nc, -1) * w[:, None]
                m = torch.nn.functional.pad(m, (0, -m.shape[1] % chunk)).reshape(nc, -1, chunk)
                need[r] = m.transpose(0, 1).contiguous()  # [chunks, nc, chunk]
        kept |= need
        a, b, c = need[r1], need[r2], need[r3]
        for p in np.flatnonzero(live):
            p0, p1 = max(0, p - n), min(nc, p + n + 1)
            x = a[:, p:p + 1] * b[:, p0:p1]
            s = torch.bmm(x, c[:, p0:p1].transpose(1, 2)).sum(0)
            out[t, p0 - p + n:p1 - p + n, p0 - p + n:p1 - p + n] += s
    return out


def normalised(gv, counts):
    seen = counts > 0
    return torch.where(seen, gv / counts.clamp(min=1.0), gv), seen.to(torch.float64)


def triplet_counts(case, ntri):
    """Channel triplets per lag cell, whole numbers, for every triangle."""
    nc, n = case["nc"], case["nc10"]
    w = np.concatenate([np.zeros(n), weights(case), np.zeros(n)])
    win = np.stack([w[p:p + 2 * n + 1] for p in range(nc)]) * weights(case)[:, None]
    one = np.rint(win.T @ np.stack([w[p:p + 2 * n + 1] for p in range(nc)])).astype(np.int64)
    return np.broadcast_to(one, (ntri, *one.shape))


def calcr_rows(case, mask):
    lo, hi = edges(case)
    maps = [planes(mask[:, :, 5:6], lo[r], hi[r], case["nn"])[0] for r in range(len(lo))]
    return np.array([[r1, r2, r3, float((maps[r1] * maps[r2] * maps[r3]).sum())] for r1, r2, r3 in closed(case)])


def too_long(case):
    return products(case) > 2.5e13


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        return exact_grid(case, seed)
    if kind == "ensemble":
        if sum(products(c) for c in mix(case)) > 2.5e13:
            return None
        return [exact_realisation(c, 17 * seed + i) for i, c in enumerate(mix(case))]
    if kind == "realisation":
        return None if too_long(case) else exact_realisation(case, seed)
    grid, mask = normalised(*cube(case, seed))
    if kind == "maps":
        return exact_maps(case, grid, mask)
    if too_long(case):
        return None
    tri = chosen(case)
    d = lag_sums(case, grid, tri)
    i = lag_sums(case, mask, tri) if case["version"] == 2 else None
    if kind == "cylbs":
        return exact_cylbs(case, d, i)
    if kind == "triangles":
        return [d, None, i]
    _, hi = edges(case)
    ng = side_of(hi[tri[0][0]])
    if case["version"] == 2:
        return [1.0 / (ng * ng), d[0], i[0]]
    num = (ng / case["nn"]) ** 2 * 1.0e6
    return [num / (ng * ng), num, d[0], None]


def exact_realisation(case, seed):
    grid, mask = normalised(*cube(case, seed))
    tri = closed(case)
    n2 = (2 * case["nc10"] + 1) ** 2
    shape = (len(tri), n2) if case.get("kind") != "realisation" else (len(tri), 2 * case["nc10"] + 1,
                                                                      2 * case["nc10"] + 1)
    out = [calcr_rows(case, mask), lag_sums(case, grid, tri).reshape(shape), None]
    return out + ([lag_sums(case, mask, tri).reshape(shape)] if case["version"] == 2 else [])


def exact_maps(case, grid, mask):
    nn, nc, bins = case["nn"], case["nc"], case["bins"]
    h = nn // 2 + 1
    umin, umax = 1.0, 0.5 * DU * nn
    size = math.log10(umax / umin) / bins
    members = [[] for _ in range(bins)]
    for i in range(nn):
        a = nn - i if i > nn // 2 else i
        for j in range(h):
            u = math.sqrt(a * a + j * j) * DU
            if umin <= u < umax:
                b = math.floor(math.log10(u / umin) / size)
                if 0 <= b < bins:
                    members[b].append((i * h + j, u))
    flat, m = grid.reshape(-1, nc), mask.reshape(-1, nc)
    cl = torch.zeros(bins, nc, dtype=torch.float64, device=grid.device)
    binu = np.zeros(bins)
    for b, cells in enumerate(members):
        if not cells:
            continue
        at = torch.tensor([c for c, _ in cells], device=grid.device)
        u = torch.tensor([v for _, v in cells], dtype=torch.float64, device=grid.device)
        g, k = flat[at], m[at]
        no = k.sum(0)
        s = (g.real * k).T @ g.real + (g.imag * k).T @ g.imag
        s = torch.where(no[:, None] > 0, s / no.clamp(min=1.0)[:, None], s)
        for d in range(nc):
            cl[b, d] = torch.diagonal(s, d).sum()
        last = float(no[-1])
        binu[b] = float((u * k[:, -1]).sum()) / (last if last else 1.0)
    return {"cldnu": cl, "numdnu": np.arange(nc, 0, -1).astype(np.float64), "binu": binu, "num": None}


def exact_cylbs(case, d, i):
    n, cut = case["nc10"], case["n_cut"]
    k = amber_b200.reference_cylbs_constants()

    def fold(a):
        low, up = a[:, :n + 1].flip(1, 2), a[:, n:]
        out = up.clone()
        out[:, 1:] += low[:, 1:]
        return out

    den = i if i is not None else torch.as_tensor(triplet_counts(case, len(d)).astype(np.float64), device=d.device)
    t = fold(d) / k["mabs_norm"] / fold(den)
    size = 2 * n + 1 - 2 * cut
    t = t[:, :n + 1 - cut, cut:cut + size]
    if case["version"] == 2:
        x = 2.0 * math.pi * torch.arange(size, dtype=torch.float64, device=d.device) / (size - 1)
        win = 0.3635819 - 0.4891775 * torch.cos(x) + 0.1365995 * torch.cos(2 * x) - 0.0106411 * torch.cos(3 * x)
        t = t * win[size // 2:][None, :, None] * win[None, None, :]
    y = torch.fft.ifft(torch.fft.ifftshift(t, dim=2).to(torch.complex128), dim=2)
    y[:, 0] = y[:, 0].real.to(y.dtype)
    out = torch.fft.irfft(y, n=size, dim=1)
    scale = k["rc"] ** 4 * (size * k["dnu_mhz"] * k["rc_prime"]) ** 2
    return torch.fft.fftshift(out, dim=(1, 2)) * scale


def exact_grid(case, seed):
    randpar, data, umax = records(case, seed)
    nn, nc, h = case["nn"], case["nc"], case["nn"] // 2 + 1
    sign = np.where(randpar[:, 1] < 0, np.float32(-1), np.float32(1)).astype(np.float32)
    nu = np.float32(NU0) * sign
    u, v = nu * randpar[:, 0], nu * randpar[:, 1]
    keep = np.sqrt((u * u + v * v).astype(np.float64)) <= umax

    def nearest(x):
        y = x.astype(np.float64) / DU
        return np.where(y < 0, -np.floor(-y + 0.5), np.floor(y + 0.5)).astype(np.int64)

    cell = torch.as_tensor((nearest(u) % nn) * h + nearest(v))[torch.as_tensor(keep)]
    d = torch.as_tensor(data[keep, :, 0]).to(torch.float64)
    live = (d[:, :, 2] > 0).to(torch.float64) if case["flag_key"] else torch.ones_like(d[:, :, 2])
    s = torch.as_tensor(sign[keep]).to(torch.float64)[:, None]
    sums = [torch.zeros(nn * h, nc, dtype=torch.float64).index_add_(0, cell, x)
            for x in (d[:, :, 0] * live, d[:, :, 1] * s * live, live)]
    k = case["collapse"]
    sums = [x[:, :nc // k * k].reshape(nn, h, nc // k, k).sum(3) for x in sums]
    return [torch.complex(sums[0], sums[1]).numpy(), sums[2].numpy()]

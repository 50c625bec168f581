"""Workloads of the fitness library, through its public entry points.

Every case evaluates compound-prism designs drawn over the synthetic optimizer's parameter
ranges (2 to 6 prisms, alternating face angles of 0.1 to 1.2 rad, curvature 0.01 to 0.1,
16 to 128 detector bins; `generations.py` and `workload.py` of the package). Each state has
its own designs, wavelengths and sampling seed. The kinds of call:

  single   Spectrometer.gpu_fitness_full, one design per call (gpu_fitness with its record)
  loop     a generation evaluated as the reference optimizer does: one gpu_fitness call per
           design, each with a random seed of its own
  points   Spectrometer.gpu_fitness_points with p(d|lambda) returned
  batch    fitness_batch on built designs
  params   fitness_batch_params: parameter records, designs built on the GPU
  server   Server.submit and wait, one generation per request
  tp       Spectrometer.transmission_probability
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "compound-prism-designer_gb300"))

WAVELENGTHS = (0.5, 0.82)  # um
WIDTH, BEAM_WIDTH = 7.0, 2.0
BINS = (16, 32, 64, 128)
ALPHA = 1.0 / 1.61803398874989484820458683436563
SEM = 5e-3
KINDS = ("single", "loop", "points", "batch", "params", "server", "tp")


# ------------------------------------------------------------------ the cases

def _case(name, kind, n, G, B, W, R, seeds=1, adaptive=False, ar=True):
    """n designs of G prisms and B bins (0: mixed), W wavelengths (0: 512 to 4096, mixed) x R rays."""
    c = {"kind": kind, "n": n, "G": G, "B": B, "W": W, "R": R, "seeds": seeds, "adaptive": adaptive, "ar": ar}
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # the smallest configuration the repository measures: a quick look at one design
        _case("single_small", "single", 1, 3, 32, 64, 256),
        # the reference optimizer's call (designer.py): one design, 128 x 8192
        _case("single_optimizer", "single", 1, 4, 64, 128, 8192),
        # the same call with the reference kernel's per-wavelength stop
        _case("single_adaptive", "single", 1, 5, 32, 128, 8192, adaptive=True),
        # gpu_fitness's default arguments, two seeds, a prism without coating
        _case("single_default_uncoated", "single", 1, 3, 64, 256, 16384, seeds=2, ar=False),
        # the repository's headline call: 6 prisms, 64 bins, 4096 x 1024
        _case("single_headline", "single", 1, 6, 64, 4096, 1024),
        # p(d|lambda) of one design on a caller's own points: plots and studies, ragged sizes
        _case("points_ragged", "points", 1, 5, 100, 1001, 3001),
        # a generation evaluated call by call, a fresh random seed for each design
        _case("loop_generation", "loop", 128, 0, 0, 128, 8192),
        # a population with mixed sampling in one call
        _case("batch_mixed", "batch", 1024, 0, 0, 0, 1024),
        # a generation of 256 with the reference kernel's per-wavelength stop
        _case("batch_adaptive", "batch", 256, 0, 0, 128, 8192, adaptive=True),
        # a generation as parameter records: built, positioned and evaluated on the GPU
        _case("params_generation", "params", 512, 0, 0, 128, 8192),
        # serving: a generation of 1024 built designs as one request
        _case("server_generation", "server", 1024, 0, 0, 128, 8192),
        # the interactive viewer's plot: p(d|lambda) at 100 wavelengths by the reference's estimator
        _case("tp_plot", "tp", 1, 4, 64, 100, 16384),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(KINDS)
    G = rng.randint(1, 6)
    ar = rng.random() < 0.8
    adaptive = kind in ("single", "batch", "params", "server") and rng.random() < 0.25
    if kind == "single":
        W = _log_int(rng, 48, 4096)
        return _case(None, kind, 1, G, _log_int(rng, 8, 256), W, _log_int(rng, 200, min(16384, (1 << 22) // W)),
                     seeds=rng.randint(1, 3), adaptive=adaptive, ar=ar)
    if kind == "loop":
        return _case(None, kind, _log_int(rng, 8, 128), 0, 0, _log_int(rng, 64, 256), _log_int(rng, 1024, 8192), ar=ar)
    if kind == "points":
        W = _log_int(rng, 60, 4096)
        return _case(None, kind, 1, G, _log_int(rng, 8, 256), W, _log_int(rng, 200, min(16384, (1 << 22) // W)), ar=ar)
    if kind == "tp":
        return _case(None, kind, 1, G, _log_int(rng, 8, 128), _log_int(rng, 10, 400), _log_int(rng, 1000, 16384), ar=ar)
    n = _log_int(rng, 16, 768)
    if rng.random() < 0.4:
        return _case(None, kind, n, 0, 0, 0, _log_int(rng, 256, 1024), adaptive=adaptive, ar=ar)
    return _case(None, kind, n, 0, 0, _log_int(rng, 64, 256), _log_int(rng, 1024, 8192), adaptive=adaptive, ar=ar)


# ------------------------------------------------------------------ the designs (f64, on the host)

def _glasses(rng, n):
    """n synthetic glasses: Sellmeier curves fitted by a degree-5 polynomial, highest degree first."""
    x = np.linspace(*WAVELENGTHS, 100)
    fit = np.linalg.pinv(np.vander(x, 6))
    b1, b2, b3 = rng.uniform(0.5, 1.8, n), rng.uniform(0.0, 0.5, n), rng.uniform(0.5, 1.5, n)
    c1, c2, c3 = rng.uniform(0.003, 0.015, n), rng.uniform(0.01, 0.07, n), rng.uniform(80, 200, n)
    w2 = (x * x)[None, :]
    s = [b[:, None] * w2 / (w2 - c[:, None]) for b, c in ((b1, c1), (b2, c2), (b3, c3))]
    return np.sqrt(1 + s[0] + s[1] + s[2]) @ fit.T


def _surfaces(D, G):
    """Adds the surfaces of designs with G prisms each to their parameters (arrays over designs)."""
    a, h2 = D["angles"], D["height"] * 0.5
    nx, ny = -np.cos(a), -np.sin(a)
    off = np.abs(ny / nx) * h2[:, None]
    px = [off[:, 0]]
    for k in range(1, G + 1):
        turn = np.signbit(ny[:, k - 1]) != np.signbit(ny[:, k])
        px.append(px[-1] + np.where(turn, off[:, k - 1] + off[:, k], np.abs(off[:, k - 1] - off[:, k])))
    D["px"], D["nx"], D["ny"], D["h2"] = np.stack(px, 1), nx, ny, h2
    k = D["curvature"]
    chord = np.abs(D["height"] / nx[:, G])
    D["rad"] = chord * 0.5 / np.abs(k)
    apothem = np.sqrt(D["rad"] ** 2 - chord ** 2 * 0.25)
    sag = D["rad"] - apothem
    ca, sa = np.copysign(apothem, k), np.copysign(sag, k)
    D["cx"], D["cy"] = nx[:, G] * ca + px[G], ny[:, G] * ca + h2
    D["mx"], D["my"] = px[G] - nx[:, G] * sa, h2 - ny[:, G] * sa
    D["rho2"] = sag ** 2 + chord ** 2 * 0.25
    return D


def _index(c, lam):
    s = c[0]
    for i in range(1, 6):
        s = s * lam + c[i]
    return s


def _prism(xp, d, G, lam, y, ar):
    """Rays (wavelength lam, start height y) through the prism: (ok, point, direction, t_s, t_p)."""
    zero = lam * 0.0 + y * 0.0
    ox, oy, dx, dy = zero, zero + y, lam * 0.0 + 1.0, lam * 0.0
    ts = tp = lam * 0.0 + 1.0
    ok = zero == 0.0

    def refract(dx, dy, ts, tp, nx, ny, n1, n2):
        ci = -(dx * nx + dy * ny)
        r = n1 / n2
        c2 = 1.0 - r * r * (1.0 - ci * ci)
        cr = xp.sqrt(xp.where(c2 > 0, c2, c2 * 0.0))
        k = r * ci - cr
        fs, fp = n1 * ci + n2 * cr, n1 * cr + n2 * ci
        rs, rp = ((n1 * ci - n2 * cr) / fs) ** 2, ((n1 * cr - n2 * ci) / fp) ** 2
        coat = (ci > 0.5) & ar
        qs, qp = xp.where(coat, ci * 0.0 + 0.99, 1.0 - rs), xp.where(coat, ci * 0.0 + 0.99, 1.0 - rp)
        return c2 >= 0, dx * r + nx * k, dy * r + ny * k, ts * qs, tp * qp

    n1 = lam * 0.0 + 1.0
    for k in range(G):
        n2 = _index(d["glass"][k], lam)
        nx, ny = d["nx"][k], d["ny"][k]
        s = ((d["px"][k] - ox) * nx + (d["h2"] - oy) * ny) / (dx * nx + dy * ny)
        ox, oy = ox + dx * s, oy + dy * s
        ok = ok & (s >= 0) & (oy >= 0) & (oy <= d["height"])
        good, dx, dy, ts, tp = refract(dx, dy, ts, tp, nx, ny, n1, n2)
        ok = ok & good
        n1 = n2
    ex, ey = ox - d["cx"], oy - d["cy"]
    ud = dx * ex + dy * ey
    disc = ud * ud - (ex * ex + ey * ey) + d["rad"] ** 2
    sd = xp.sqrt(xp.where(disc > 0, disc, disc * 0.0))

    def inside(s):
        qx, qy = ox + dx * s - d["mx"], oy + dy * s - d["my"]
        return (s >= 0) & (qx * qx + qy * qy <= d["rho2"])

    s1, s2 = -ud - sd, sd - ud
    first = inside(s1)
    s = xp.where(first, s1, s2)
    ok = ok & (disc > 0) & (first | inside(s2))
    ox, oy = ox + dx * s, oy + dy * s
    good, dx, dy, ts, tp = refract(dx, dy, ts, tp, (d["cx"] - ox) / d["rad"], (d["cy"] - oy) / d["rad"], n1,
                                   n1 * 0.0 + 1.0)
    return ok & good, ox, oy, dx, dy, ts, tp


def _place(D, G, ar):
    """Places each design's detector where the axial rays of both ends of the wavelength range meet
    its two ends. Adds `pos`, `flipped`; returns which designs can be placed."""
    d = {k: D[k] for k in ("height", "cx", "cy", "rad", "mx", "my", "rho2", "h2")}
    for k in ("px", "nx", "ny"):
        d[k] = [D[k][:, i] for i in range(D[k].shape[1])]
    d["glass"] = [[D["glass"][:, k, i] for i in range(6)] for k in range(G)]
    ends = [_prism(np, d, G, np.full(len(D["height"]), w), D["y_mean"], ar) for w in WAVELENGTHS]
    (ok0, x0, y0, u0, v0, s0, p0), (ok1, x1, y1, u1, v1, s1, p1) = ends
    sx, sy = -np.sin(D["det_angle"]) * 32.0, np.cos(D["det_angle"]) * 32.0
    det = u1 * -v0 + u0 * v1

    def along(sign):
        tx, ty = sign * sx - x1 + x0, sign * sy - y1 + y0
        return -v1 / det * tx + u1 / det * ty

    up, down = along(1.0), along(-1.0)
    dist = np.where(up > 0, up, down)
    D["flipped"] = ~(up > 0)
    D["pos"] = np.stack([x0 + u0 * dist, y0 + v0 * dist], 1)
    return ok0 & ok1 & (s0 + p0 > 2e-2) & (s1 + p1 > 2e-2) & (np.abs(det) > 1e-9) & (dist > 1e-9)


def _designs(rng, case):
    """The case's designs as a list of dicts of plain f64 values (draws that cannot be placed are redrawn)."""
    n = case["n"]
    Gs = np.full(n, case["G"]) if case["G"] else rng.integers(2, 7, n)
    Bs = np.full(n, case["B"]) if case["B"] else rng.choice(BINS, n)
    out = [None] * n
    with np.errstate(all="ignore"):
        for G in sorted(set(Gs.tolist())):
            want = np.nonzero(Gs == G)[0]
            got = 0
            while got < want.size:
                m = 8 * (want.size - got) + 32
                D = {"glass": _glasses(rng, m * G).reshape(m, G, 6),
                     "angles": np.where(rng.uniform(size=(m, 1)) < 0.5, 1.0, -1.0) * (-1.0) ** np.arange(G + 1)
                     * rng.uniform(0.1, 1.2, (m, G + 1)),
                     "curvature": rng.uniform(0.01, 0.1, m), "height": rng.uniform(15.0, 25.0, m),
                     "det_angle": rng.uniform(-0.6, 0.6, m)}
                D["y_mean"] = D["height"] * rng.uniform(0.3, 0.7, m)
                ok = _place(_surfaces(D, G), G, case["ar"])
                for i in np.nonzero(ok)[0][: want.size - got]:
                    B = int(Bs[want[got]])
                    out[want[got]] = dict({k: v[i] for k, v in D.items()}, G=G, B=B, slope=32.0 / B,
                                          ar=case["ar"])
                    got += 1
    return out


def _sampling(rng, case):
    n = case["n"]
    W = np.full(n, case["W"]) if case["W"] else rng.integers(512, 4097, n)
    return W.astype(np.int64), np.full(n, case["R"], dtype=np.int64)


def _inputs(case, seed):
    rng = np.random.default_rng([20261205, int(seed)])
    ds = _designs(rng, case)
    W, R = _sampling(rng, case)
    if case["kind"] == "loop":
        seeds = rng.uniform(size=case["n"])
    else:
        seeds = rng.uniform(size=max(1, case["seeds"]))
    return ds, W, R, seeds


# ------------------------------------------------------------------ prepare and run

def _spectrometer(cpd, d):
    glasses = [cpd.Glass("g%d" % i, c) for i, c in enumerate(d["glass"])]
    prism = cpd.CompoundPrism(glasses, d["angles"], [0.0] * d["G"], float(d["curvature"]), float(d["height"]), WIDTH,
                              bool(d["ar"]))
    wl = cpd.UniformWavelengthDistribution(WAVELENGTHS)
    beam = cpd.GaussianBeam(BEAM_WIDTH, float(d["y_mean"]))
    s = d["slope"]
    det = cpd.DetectorArray(d["B"], 0.8 * s, s, 0.1 * s, 32.0, math.radians(45.0), float(d["det_angle"]),
                            (float(d["pos"][0]), float(d["pos"][1])), bool(d["flipped"]))
    spec = cpd.Spectrometer(prism, det, wl, beam)
    _ = spec.design
    return spec


def _records(N, ds):
    p = np.zeros(len(ds), dtype=N.PARAMS_DTYPE)
    for r, d in zip(p, ds):
        G = d["G"]
        r["nglass"], r["ar_coated"] = G, int(d["ar"])
        r["glass"][:G] = d["glass"]
        r["angles"][: G + 1] = d["angles"]
        r["curvature"], r["height"], r["width"] = d["curvature"], d["height"], WIDTH
        r["bin_count"], r["bin_size"] = d["B"], 0.8 * d["slope"]
        r["linear_slope"], r["linear_intercept"] = d["slope"], 0.1 * d["slope"]
        r["det_length"], r["max_incident_angle"], r["det_angle"] = 32.0, math.radians(45.0), d["det_angle"]
        r["det_position"], r["det_flipped"] = d["pos"], int(d["flipped"])
        r["wavelength_bounds"] = WAVELENGTHS
        r["beam_width"], r["beam_y_mean"] = BEAM_WIDTH, d["y_mean"]
    return p


def _points(seed, first, n):
    v = np.arange(first, first + n) * ALPHA + seed
    return v - np.trunc(v)


def prepare(case, seed):
    import compound_prism_designer as cpd
    from compound_prism_designer import _native as N

    kind = case["kind"]
    ds, W, R, seeds = _inputs(case, seed)
    st = {"cpd": cpd, "kind": kind, "adaptive": case["adaptive"], "ctx": cpd.default_context(),
          "mode": cpd.TRACE_HYBRID | (cpd.SAMPLING_ADAPTIVE if case["adaptive"] else 0),
          "W": int(W[0]), "R": int(R[0]), "seeds": [float(s) for s in seeds]}
    if kind == "params":
        st.update(params=_records(N, ds), Ws=W, Rs=R)
    elif kind == "server":
        designs, status = cpd.build_designs(_records(N, ds))
        assert not status.any()
        st.update(designs=designs, Ws=W, Rs=R, server=cpd.Server())
    else:
        specs = [_spectrometer(cpd, d) for d in ds]
        st.update(specs=specs, spec=specs[0], Ws=W, Rs=R)
        if kind == "points":
            st.update(lam=_points(seeds[0], 0, st["W"]), rays=_points(seeds[0], 1, st["R"]))
        if kind == "tp":
            lo, hi = WAVELENGTHS
            st["wavelengths"] = lo + (hi - lo) * (np.arange(st["W"]) + seeds[0]) / st["W"]
    return st


def _of_record(f):
    return {"info": f.info, "size": f.size, "deviation": f.deviation, "h_cond": f.h_cond, "h_det": f.h_det,
            "max_sem": f.max_sem, "rays": f.rays, "hits": f.hits, "wavelengths": f.wavelengths, "status": f.status}


def _of_array(o):
    return {"info": o["info"], "size": o["size"], "deviation": o["deviation"], "rays": o["rays"].astype(np.int64),
            "hits": o["hits"].astype(np.int64), "status": o["status"]}


def run(state):
    s, kind, cpd = state, state["kind"], state["cpd"]
    if kind == "single":
        return _of_record(s["spec"].gpu_fitness_full(s["seeds"], max_n=s["W"], max_eval=s["R"],
                                                     adaptive=s["adaptive"]))
    if kind == "loop":
        fs = [spec.gpu_fitness_full([seed], max_n=s["W"], max_eval=s["R"])
              for spec, seed in zip(s["specs"], s["seeds"])]
    elif kind == "points":
        f, p = s["spec"].gpu_fitness_points(s["lam"], s["rays"], want_p=True)
        return dict(_of_record(f), p=p)
    elif kind == "tp":
        return dict(zip(("p", "rays"), s["spec"].transmission_probability(s["wavelengths"], max_m=s["R"],
                                                                          return_rays=True)))
    elif kind == "batch":
        fs = cpd.fitness_batch(s["specs"], seeds=s["seeds"][0], max_n=s["Ws"], max_eval=s["Rs"], mode=s["mode"])
    elif kind == "params":
        return _of_array(cpd.fitness_batch_params(s["params"], acceptance=1.0, seeds=s["seeds"][0], max_n=s["Ws"],
                                                  max_eval=s["Rs"], mode=s["mode"]))
    else:
        rid = s["server"].submit(s["designs"], seeds=s["seeds"][0], max_n=s["Ws"], max_eval=s["Rs"], mode=s["mode"])
        return _of_array(s["server"].wait(rid)[0])
    return {"info": np.array([f.info for f in fs]), "size": np.array([f.size for f in fs]),
            "deviation": np.array([f.deviation for f in fs]), "rays": np.array([f.rays for f in fs]),
            "hits": np.array([f.hits for f in fs]), "status": np.array([f.status for f in fs])}


def work(case):
    """Each design's record read and its result written once; per wavelength one chain through the flat
    faces (39 FLOP each), per ray the exit face and the detector (82 FLOP)."""
    G = case["G"] or 4
    W = case["W"] or 2304
    B = case["B"] or 60
    rows = case["n"] * W * (case["seeds"] if case["kind"] == "single" else 1)
    out = 8 * W * B if case["kind"] in ("points", "tp") else 0
    return {"bytes": case["n"] * (1200 + 96) + out, "flops": float(rows) * (39 * G + 82 * case["R"])}


# ------------------------------------------------------------------ the same in 64 bits

def _norminv(u):
    """Shaw's rational approximation of the inverse normal CDF (arXiv:0901.0638)."""
    P = (4.3304513840364031401e-8, 0.000036313870818023761224, 0.0034424140686962222423, 0.085838533424158257377,
         0.73176759583280610539, 2.3884158540184385711, 3.0333178251950406994, 1.2533141359896652729)
    Q = (1.3141263119543315917e-6, 0.00030617264753008793976, 0.014494272424798068406, 0.2168237095066675527,
         1.2356513216582148689, 2.9373357991677046357, 2.9202373175993672857, 1.0)
    v = -np.log(2.0 * np.where(u > 0.5, 1.0 - u, u))
    return np.copysign(v * np.polyval(P, v) / np.polyval(Q, v), u - 0.5)


def _rays(d, lam, z, dev):
    """(bin or B where lost, t) of every (wavelength, start height) pair."""
    T = lambda v: torch.as_tensor(np.asarray(v, dtype=np.float64), device=dev)  # noqa: E731
    G = d["G"]
    s = {k: float(d[k]) for k in ("height", "cx", "cy", "rad", "mx", "my", "rho2", "h2")}
    s.update({k: [float(v) for v in d[k]] for k in ("px", "nx", "ny")})
    s["glass"] = [[float(v) for v in g] for g in d["glass"]]
    y = float(d["y_mean"]) - BEAM_WIDTH * T(z)[None, :]
    ok, ox, oy, dx, dy, ts, tp = _prism(torch, s, G, T(lam)[:, None], y, bool(d["ar"]))
    a = float(d["det_angle"])
    nx, ny = -math.cos(a), -math.sin(a)
    ux, uy = (-ny, nx) if d["flipped"] else (ny, -nx)
    ci = -(dx * nx + dy * ny)
    px, py = ox - float(d["pos"][0]), oy - float(d["pos"][1])
    dist = (px * nx + py * ny) / ci
    pos = (px + dx * dist) * ux + (py + dy * dist) * uy
    q = torch.floor((pos - 0.1 * d["slope"]) / d["slope"])
    rem = pos - 0.1 * d["slope"] - q * d["slope"]
    ok = ok & (ci > math.cos(math.radians(45.0))) & (pos >= 0) & (pos <= 32.0) & (rem < 0.8 * d["slope"]) & (q < d["B"])
    # a bin index below zero saturates to bin 0
    return torch.where(ok, q.clamp(min=0.0), q * 0.0 + d["B"]).nan_to_num(nan=float(d["B"])).long(), (ts + tp) * 0.5


def _sums(b, t, B):
    """Sum of t per (wavelength, bin)."""
    W = b.shape[0]
    idx = torch.arange(W, device=b.device)[:, None] * (B + 1) + b
    h = torch.zeros(W * (B + 1), dtype=torch.float64, device=b.device)
    h.index_add_(0, idx.reshape(-1), (t + torch.zeros_like(b, dtype=t.dtype)).reshape(-1))
    return h.reshape(W, B + 1)[:, :B]


def _adaptive_sums(b, t, B):
    """p(d|lambda) when each wavelength stops after the first round of 32 rays that hit some bin and after
    which every bin it hit has SEM below 5e-3 (a bin's samples are those of the rounds that hit it)."""
    W, R = b.shape
    rounds = (R + 31) // 32
    rnd = torch.arange(R, device=b.device) // 32
    idx = (torch.arange(W, device=b.device)[:, None] * rounds + rnd[None, :]) * (B + 1) + b
    t = t + torch.zeros_like(b, dtype=torch.float64)

    def cells(v):
        h = torch.zeros(W * rounds * (B + 1), dtype=torch.float64, device=b.device)
        return h.index_add_(0, idx.reshape(-1), v.reshape(-1)).reshape(W, rounds, B + 1)[:, :, :B]

    hit = cells(torch.ones_like(t)) > 0
    size = torch.clamp(R - 32 * torch.arange(rounds, device=b.device), max=32).double()
    n = (hit * size[None, :, None]).cumsum(1)
    s1, s2 = cells(t).cumsum(1), cells(t * t).cumsum(1)
    good = (s2 - s1 * s1 / n.clamp(min=1.0)) < SEM * SEM * n * (n - 1)
    stop = hit.any(2) & (good | ~hit).all(2)
    last = torch.where(stop.any(1), stop.double().argmax(1), torch.full((W,), rounds - 1, device=b.device))
    used = torch.clamp((last + 1) * 32, max=R).double()
    return s1.gather(1, last[:, None, None].expand(W, 1, B))[:, 0] / used[:, None]


def _plogp(p):
    return torch.where(p > 0, p * torch.log2(p.clamp(min=1e-300)), p * 0.0)


def _p_of(case, d, lam_u, ray_u, dev):
    z = _norminv(ray_u)
    lo, hi = WAVELENGTHS
    out, step = [], max(1, (1 << 23) // max(1, z.size))
    for k in range(0, lam_u.size, step):
        b, t = _rays(d, lo + (hi - lo) * lam_u[k: k + step], z, dev)
        out.append(_adaptive_sums(b, t, d["B"]) if case["adaptive"] else _sums(b, t, d["B"]) / z.size)
    return torch.cat(out)


def _summary(d, p):
    n = p.shape[0]
    h_cond, h_det = float(_plogp(p).sum(1).mean()), float(_plogp(p.mean(0)).sum())
    m2 = ((p - p.mean(0)) ** 2).sum(0)
    a = float(d["det_angle"])
    nx, ny = -math.cos(a), -math.sin(a)
    ux, uy = (-ny, nx) if d["flipped"] else (ny, -nx)
    x, y = float(d["pos"][0]) + 16.0 * ux, float(d["pos"][1]) + 16.0 * uy - float(d["y_mean"])
    size = math.hypot(x, y)
    return {"info": h_cond - h_det, "size": size, "deviation": abs(y / size), "h_cond": h_cond, "h_det": h_det,
            "max_sem": math.sqrt(float((m2 / max(1, n - 1) / n).max())),
            "converged": bool((m2 < SEM * SEM * n * (n - 1)).all())}


def _tp(d, lam, R, dev):
    """The reference's estimator, ray by ray for all wavelengths: a hit pads its bin's running mean and squared
    deviations with zeros up to the ray count (with the padded mean in the deviations' update, as the reference has
    it) and adds its t; the wavelength stops at the first hit whose bin's SEM is below 5e-3; every bin is then
    padded to the final count."""
    u = (0.5 + np.arange(1, R + 1) * ALPHA) % 1.0
    b, t = _rays(d, lam, _norminv(u), dev)
    b, t = b.cpu().numpy(), (t + torch.zeros_like(b, dtype=torch.float64)).cpu().numpy()
    W, B = b.shape[0], d["B"]
    c, m, m2 = np.zeros((W, B)), np.zeros((W, B)), np.zeros((W, B))
    count = np.full(W, float(R))
    live = np.ones(W, dtype=bool)
    for j in range(R):
        i = np.nonzero(live & (b[:, j] < B))[0]
        if i.size == 0:
            if not live.any():
                break
            continue
        k, v, n = b[i, j], t[i, j], j + 1.0
        ci, mi, qi = c[i, k], m[i, k], m2[i, k]
        pad = ci < n
        mp = np.where(pad, ci * mi / n, mi)
        qi = np.where(pad, qi + mp * mp * ci * (n - ci) / n, qi)
        ci = np.maximum(ci, n) + 1.0
        dv = v - mp
        mi = mp + dv / ci
        qi = qi + dv * (v - mi)
        c[i, k], m[i, k], m2[i, k] = ci, mi, qi
        done = i[qi < SEM * SEM * (ci * (ci - 1.0))]
        live[done] = False
        count[done] = n
    n = count[:, None]
    return np.where(c < n, c * m / n, m)


def exact(case, seed):
    n, kind = case["n"], case["kind"]
    ds, W, R, seeds = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rays = float((W * R).sum()) * (case["seeds"] if kind == "single" else 1)
    if rays > (3e9 if dev == "cuda" else 2e7):
        return None
    if kind == "tp":
        lo, hi = WAVELENGTHS
        lam = lo + (hi - lo) * (np.arange(int(W[0])) + seeds[0]) / int(W[0])
        return {"p": _tp(ds[0], lam, int(R[0]), dev), "rays": None}
    keys = ("info", "size", "deviation")
    if kind in ("single", "points"):
        ps = []
        for s in seeds:
            ps.append(_p_of(case, ds[0], _points(s, 0, int(W[0])), _points(s, 1, int(R[0])), dev))
            o = _summary(ds[0], torch.cat(ps))
            if o["converged"] or kind == "points":
                break
        r = {k: o[k] for k in keys + ("h_cond", "h_det", "max_sem")}
        r.update(rays=None, hits=None, wavelengths=None, status=None)
        if kind == "points":
            r["p"] = ps[0].cpu().numpy()
        return r
    each = [seeds[i] if kind == "loop" else seeds[0] for i in range(n)]
    os_ = [_summary(d, _p_of(case, d, _points(s, 0, int(w)), _points(s, 1, int(r)), dev))
           for d, s, w, r in zip(ds, each, W, R)]
    return dict({k: np.array([o[k] for o in os_]) for k in keys}, rays=None, hits=None, status=None)

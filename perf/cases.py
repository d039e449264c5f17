"""Timed cases of the time-step library, over the range its users run.

A pass is what a program does between two frames: steps of a scene through the
public entry points, then the frame read back into page-locked arrays. Every
scene starts from a state in motion (a column under its own weight with a
velocity field and strain scatter, a pile under contact load), made from the
seed, and a further pass continues from where the last one ended.

``exact`` evaluates the same steps in 64 bits with plain torch operations.
"""
import math

import numpy as np
import torch

import libhybridgrains_gb300 as hg

GRAVITY = (0.0, -9.81)
RHO, YOUNG, POISSON = 1550.0, 1.0e6, 0.3
SHEAR = YOUNG / (2.0 * (1.0 + POISSON))
BULK = YOUNG / (3.0 * (1.0 - 2.0 * POISSON))
FLIP = 0.999
DISK_RHO = 2600.0
KN, MU_DISK = 1.0e5, 0.5
EXACT_SECONDS = 15.0


def listed():
    return [
        # the 12,800-point column a CPU user runs, 100 steps between frames
        dict(name="mpm_mixed_12800", kind="mpm", precision="mixed", basis="linear", h=5.0e-3,
             nx=200, ny=100, x0=20, wc=40, hc=80, phi=30.0, steps=100, per_call=100),
        # the large single-GPU column
        dict(name="mpm_mixed_2m", kind="mpm", precision="mixed", basis="linear", h=1.0e-3,
             nx=2048, ny=1024, x0=0, wc=1000, hc=500, phi=30.0, steps=64, per_call=64),
        # the uGIMP basis on an odd-sized column and grid
        dict(name="mpm_mixed_ugimp_611k", kind="mpm", precision="mixed", basis="ugimp", h=1.0e-3,
             nx=1371, ny=533, x0=3, wc=503, hc=304, phi=25.0, steps=48, per_call=48),
        # the drop-in loop that keeps its state in host arrays: upload, one
        # step, download
        dict(name="mpm_mixed_roundtrip_2m", kind="roundtrip", precision="mixed", basis="linear",
             h=1.0e-3, nx=2048, ny=1024, x0=0, wc=1000, hc=500, phi=30.0, steps=2, per_call=1),
        # the FP64 drop-in, one flow call per step as the reference's loop makes
        dict(name="mpm_fp64_12800", kind="mpm", precision="fp64", basis="linear", h=5.0e-3,
             nx=200, ny=100, x0=20, wc=40, hc=80, phi=30.0, steps=50, per_call=1),
        # the FP64 uGIMP bulk of the hybrid column alone
        dict(name="mpm_fp64_ugimp_100k", kind="mpm", precision="fp64", basis="ugimp", h=2.5e-3,
             nx=404, ny=404, x0=0, wc=100, hc=250, phi=30.0, steps=24, per_call=24),
        # a small pile on a row of fixed disks stepped one call at a time:
        # launches and latency
        dict(name="dem_fp64_1000", kind="dem", precision="fp64", n=1000, per_row=40,
             pitch=1.9e-3, fixed_row=True, dt=1.0e-6, steps=50, per_call=1),
        # the 10,000-disk pile under contact load, bit-exact law
        dict(name="dem_fp64_10k", kind="dem", precision="fp64", n=10000, per_row=100,
             pitch=1.9e-3, fixed_row=False, dt=1.0e-6, steps=100, per_call=100),
        # a million disks under contact load, mixed-precision law
        dict(name="dem_mixed_1m", kind="dem", precision="mixed", n=1000000, per_row=1000,
             pitch=1.9e-3, fixed_row=False, dt=1.0e-6, steps=16, per_call=16),
        # the hybrid column between two resamplings, both precisions: uGIMP
        # bulk under grains that overlap it by four cells, both fields
        # homogenised
        dict(name="hybrid_fp64", kind="hybrid", precision="fp64", wc=100, hc=250, n=8916,
             steps=20, per_call=20),
        dict(name="hybrid_mixed", kind="hybrid", precision="mixed", wc=100, hc=250, n=8916,
             steps=100, per_call=100),
        # a serving mix: small columns of 2e3 to 1e5 points stepped together
        dict(name="batch_48", kind="batch", members=48, pmin=2000, pmax=100000, sizes=7,
             steps=100, per_call=100),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _clamp(x, lo, hi):
    return int(max(lo, min(hi, x)))


def draw(rng):
    kind = rng.choice(["mpm", "mpm", "mpm64", "roundtrip", "dem", "dem", "hybrid", "batch"])
    if kind in ("mpm", "mpm64", "roundtrip"):
        fp64 = kind == "mpm64"
        cells = _log(rng, 500, 50000 if fp64 else 450000)
        aspect = rng.uniform(0.5, 4.0)
        wc = max(int(round(math.sqrt(cells / aspect))), 4)
        hc = max(int(round(cells / wc)), 4)
        h = rng.choice([1.0e-3, 2.5e-3, 5.0e-3])
        x0 = rng.randint(0, 20)
        basis = rng.choice(["linear", "ugimp"])
        points = 4 * wc * hc
        steps = _clamp(3.2e6 / points, 8, 64) if fp64 else _clamp(1.0e8 / points, 16, 100)
        if kind == "roundtrip":
            return dict(kind="roundtrip", precision="mixed", basis=basis, h=h,
                        nx=x0 + 2 * wc + rng.randint(8, 70), ny=hc + rng.randint(8, 40), x0=x0,
                        wc=wc, hc=hc, phi=rng.uniform(20.0, 40.0), steps=rng.randint(1, 2),
                        per_call=1)
        return dict(kind="mpm", precision="fp64" if fp64 else "mixed", basis=basis, h=h,
                    nx=x0 + 2 * wc + rng.randint(8, 70), ny=hc + rng.randint(8, 40), x0=x0,
                    wc=wc, hc=hc, phi=rng.uniform(20.0, 40.0), steps=steps,
                    per_call=rng.choice([1, steps, steps]))
    if kind == "dem":
        n = _log(rng, 500, 1.0e6)
        precision = rng.choice(["fp64", "mixed"])
        packed = rng.random() < 0.7
        steps = _clamp(7.0e6 / n, 6, 100)
        return dict(kind="dem", precision=precision, n=n,
                    per_row=max(int(math.sqrt(n) * rng.uniform(0.6, 1.6)), 8),
                    pitch=1.9e-3 if packed else 2.2e-3, fixed_row=rng.random() < 0.3,
                    dt=1.0e-6 if packed else 1.0e-5, steps=steps,
                    per_call=rng.choice([1, steps, steps]))
    if kind == "hybrid":
        precision = rng.choice(["fp64", "mixed"])
        s = rng.uniform(0.3, 1.0)
        return dict(kind="hybrid", precision=precision, wc=int(100 * s), hc=int(250 * s),
                    n=int(8916 * s * s * rng.uniform(0.6, 1.2)),
                    steps=rng.randint(8, 20) if precision == "fp64" else rng.randint(20, 100),
                    per_call=1000)
    steps = rng.randint(16, 100)
    return dict(kind="batch", members=_log(rng, 4, 48), pmin=2000, pmax=_log(rng, 5000, 90000),
                sizes=rng.randint(0, 999), steps=steps, per_call=steps)


# ---- scenes -----------------------------------------------------------------

def _dp_alpha(phi_deg):
    s = math.sin(math.radians(phi_deg))
    return math.sqrt(2.0 / 3.0) * 2.0 * s / (3.0 - s)


def _column(case, seed):
    """A column in motion: points, grid and planes (floor and two walls). The
    uGIMP grid goes four cells past the planes, for the points' extents."""
    h, wc, hc = case["h"], case["wc"], case["hc"]
    pad = 4 if case["basis"] == "ugimp" else 0
    rng = np.random.default_rng([int(seed), wc, hc])
    off = (np.arange(2) + 0.5) / 2.0
    gx = (np.arange(case["x0"], case["x0"] + wc)[:, None] + off).ravel()
    gy = (np.arange(hc)[:, None] + off).ravel()
    n = gx.size * gy.size
    q = np.empty((gy.size, gx.size, 2))
    q[..., 0], q[..., 1] = gx, gy[:, None]
    q = q.reshape(n, 2)
    rel = np.stack([(q[:, 0] - case["x0"]) / wc, q[:, 1] / hc], axis=1)
    q += rng.uniform(-0.1, 0.1, (n, 2))
    q *= h
    # collapse: the top moves right and down, with scatter
    v = np.empty((n, 2))
    v[:, 0] = 0.4 * rel[:, 0] * rel[:, 1]
    v[:, 1] = -0.3 * rel[:, 0] * rel[:, 1]
    v += rng.normal(0.0, 0.005, (n, 2))
    # weight of the material above, and shear strain up to the yield surface
    p = RHO * 9.81 * (1.0 - rel[:, 1]) * hc * h / BULK
    J = 1.0 - p * (1.0 + rng.uniform(-0.02, 0.02, n))
    e, s = p * rng.uniform(-0.5, 0.5, n), p * rng.uniform(-0.5, 0.5, n)
    be = np.stack([1.0 + e, s, s, (1.0 + s * s) / (1.0 + e)], axis=1)
    half = 0.25 * h
    vol = np.full(n, 4.0 * half * half)
    pts = dict(q=q, v=v, m=RHO * vol, vol=vol, hl=np.full(n, half), be=be, J=J)
    far = (case["nx"] - 2 * pad) * h
    planes = [((0.0, 0.0), (0.0, 1.0)), ((0.0, 0.0), (1.0, 0.0)), ((far, 0.0), (-1.0, 0.0))]
    lo = -pad * h
    return dict(pts=pts, planes=planes, gmin=(lo, lo), h=h, alpha=_dp_alpha(case["phi"]),
                gmax=(lo + case["nx"] * h, lo + (case["ny"] + 2 * pad) * h),
                basis=case["basis"], dt=2.0e-3 * h)


def _disks(case, seed, x0=0.0, y0=0.0, walls=True):
    """Disks of 0.9 to 1.1 mm on a jittered hex lattice; below a mean
    diameter of pitch they carry about 2.8 contacts each."""
    n, per_row, pitch = case["n"], case["per_row"], case["pitch"]
    rng = np.random.default_rng([int(seed), n, per_row])
    r = rng.uniform(0.9e-3, 1.1e-3, n)
    k = np.arange(n)
    row, col = k // per_row, k % per_row
    jit = rng.uniform(-0.05e-3, 0.05e-3, (n, 2))
    q = np.zeros((n, 3))
    q[:, 0] = x0 + pitch * (col + 0.5 + 0.5 * (row % 2)) + jit[:, 0]
    q[:, 1] = y0 + pitch * (0.5 + row * math.sqrt(3.0) / 2.0) + jit[:, 1]
    q[:, 2] = rng.uniform(-math.pi, math.pi, n)
    v = np.concatenate([rng.normal(0.0, 0.02, (n, 2)), rng.normal(0.0, 5.0, (n, 1))], axis=1)
    m = DISK_RHO * math.pi * r * r
    fixed = np.zeros(n, dtype=np.uint8)
    if case["fixed_row"]:
        fixed[:per_row] = 1
        v[:per_row] = 0.0
    planes = [((0.0, 0.0), (0.0, 1.0))]
    if walls:
        planes += [((0.0, 0.0), (1.0, 0.0)), (((per_row + 0.5) * pitch, 0.0), (-1.0, 0.0))]
    return dict(q=q, v=v, r=r, m=m, I=0.5 * m * r * r, fixed=fixed, planes=planes)


def _penalty():
    """(kn, kt, gamma_n, gamma_t, mu): normal damping for a restitution of 1/2."""
    m = DISK_RHO * math.pi * 1.0e-6
    le = math.log(0.5)
    g = 2.0 * (2.0 * math.sqrt(0.5 * m * KN) * -le / math.sqrt(math.pi ** 2 + le * le))
    return KN, 2.0 / 7.0 * KN, g, g, MU_DISK


def _hybrid_scene(case, seed):
    """The hybrid column: h = 2.5 mm, grains from four cells below the top."""
    h, wc, hc = 2.5e-3, case["wc"], case["hc"]
    col = _column(dict(h=h, wc=wc, hc=hc, x0=0, nx=4 * wc + 4, ny=2 * hc, basis="ugimp",
                       phi=30.0), seed)
    col["dt"] = 1.0e-6
    pitch = 1.95e-3
    dem = _disks(dict(n=case["n"], per_row=max(int(wc * h / pitch) - 1, 4), pitch=pitch,
                      fixed_row=False), seed, y0=(hc - 4) * h)
    dem["planes"] = col["planes"]
    return col, dem


def _batch_cases(case):
    """The members' columns: sizes and shapes fixed by the case."""
    rng = np.random.default_rng([case["sizes"], case["members"]])
    out = []
    for _ in range(case["members"]):
        cells = math.exp(rng.uniform(math.log(case["pmin"]), math.log(case["pmax"]))) / 4.0
        aspect = rng.uniform(0.5, 4.0)
        wc = max(int(round(math.sqrt(cells / aspect))), 2)
        hc = max(int(round(cells / wc)), 2)
        out.append(dict(h=5.0e-3, nx=wc + 2 * hc + 8, ny=hc + 8, x0=2, wc=wc, hc=hc,
                        basis="linear", phi=rng.uniform(20.0, 40.0)))
    return out


# ---- the library's objects --------------------------------------------------

_context = None


def _ctx():
    global _context
    if _context is None:
        _context = hg.Context(0)
    return _context


def _make_mpm(col, precision):
    n = len(col["pts"]["m"])
    return hg.MPM(_ctx(), col["gmin"], col["gmax"], col["h"], SHEAR, BULK, col["alpha"], FLIP,
                  GRAVITY, [(x, nn, True) for x, nn in col["planes"]],
                  basis=hg.UGIMP if col["basis"] == "ugimp" else hg.LINEAR,
                  precision=hg.FP64 if precision == "fp64" else hg.MIXED, capacity=n)


def _upload(m, p):
    m.upload(p["q"], p["v"], p["m"], p["vol"], p["hl"], p["be"], p["J"])


def _point_arrays(n):
    return dict(q=hg.pinned((n, 2)), v=hg.pinned((n, 2)), be=hg.pinned((n, 4)), J=hg.pinned(n))


def _make_dem(sc, precision):
    n = len(sc["r"])
    d = hg.DEM(_ctx(), GRAVITY, *_penalty(), sc["planes"], capacity=n, contact_capacity=6 * n,
               precision=hg.FP64 if precision == "fp64" else hg.MIXED)
    d.upload(sc["q"], sc["v"], sc["r"], sc["m"], sc["I"], sc["fixed"])
    return d


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind in ("mpm", "roundtrip"):
        col = _column(case, seed)
        p = col["pts"]
        s["mpm"], s["dt"] = _make_mpm(col, case["precision"]), col["dt"]
        s["out"] = _point_arrays(len(p["m"]))
        if kind == "roundtrip":
            s["const"] = {k: hg.pinned(len(p["m"])) for k in ("m", "vol", "hl")}
            for k, a in list(s["out"].items()) + list(s["const"].items()):
                a[...] = p[k]
        _upload(s["mpm"], p)
    elif kind == "dem":
        sc = _disks(case, seed)
        s["dem"], s["dt"] = _make_dem(sc, case["precision"]), case["dt"]
        s["out"] = dict(q=hg.pinned((case["n"], 3)), v=hg.pinned((case["n"], 3)))
    elif kind == "hybrid":
        col, sc = _hybrid_scene(case, seed)
        s["mpm"], s["dt"] = _make_mpm(col, case["precision"]), col["dt"]
        _upload(s["mpm"], col["pts"])
        s["dem"] = _make_dem(sc, case["precision"])
        s["hyb"] = hg.Hybrid(_ctx(), s["mpm"], s["dem"])
        nn = s["mpm"].nnodes
        s["out"] = dict(points=_point_arrays(len(col["pts"]["m"])),
                        grains=dict(q=hg.pinned((case["n"], 3)), v=hg.pinned((case["n"], 3))),
                        stress=hg.pinned((nn, 4)), velocity=hg.pinned((nn, 2)))
    else:
        cols = [_column(c, int(seed) + 1000 * i) for i, c in enumerate(_batch_cases(case))]
        ends = np.cumsum([0] + [len(c["pts"]["m"]) for c in cols])
        s["batch"] = hg.Batch(_ctx(), max_members=max(len(cols), 1))
        s["out"] = dict(q=hg.pinned((int(ends[-1]), 2)), v=hg.pinned((int(ends[-1]), 2)))
        s["members"] = []
        for c, a, b in zip(cols, ends[:-1], ends[1:]):
            m = _make_mpm(c, "mixed")
            _upload(m, c["pts"])
            s["batch"].add(m, c["dt"])
            s["members"].append((m, s["out"]["q"][a:b], s["out"]["v"][a:b]))
    return s


def _advance(step, case):
    done = 0
    while done < case["steps"]:
        k = min(case["per_call"], case["steps"] - done)
        step(k)
        done += k


def run(state):
    case, out = state["case"], state["out"]
    kind = case["kind"]
    if kind == "mpm":
        m, dt = state["mpm"], state["dt"]
        _advance(lambda k: m.flow(dt, k), case)
        m.download_into(out["q"], out["v"], out["be"], out["J"])
    elif kind == "roundtrip":
        m, c = state["mpm"], state["const"]
        for _ in range(case["steps"]):
            m.upload(out["q"], out["v"], c["m"], c["vol"], c["hl"], out["be"], out["J"])
            m.flow(state["dt"], 1)
            m.download_into(out["q"], out["v"], out["be"], out["J"])
    elif kind == "dem":
        d, dt = state["dem"], state["dt"]
        _advance(lambda k: d.flow(dt, k), case)
        d.download_into(out["q"], out["v"])
    elif kind == "hybrid":
        h, dt = state["hyb"], state["dt"]
        h.clear_homogenized()
        _advance(lambda k: h.step(dt, k, True, True), case)
        p, g = out["points"], out["grains"]
        state["mpm"].download_into(p["q"], p["v"], p["be"], p["J"])
        state["dem"].download_into(g["q"], g["v"])
        h.homogenized_into(out["stress"], out["velocity"])
    else:
        _advance(state["batch"].step, case)
        for m, q, v in state["members"]:
            m.frame_async(q, v)
    return out


# ---- what a pass cannot do without -----------------------------------------

def _mpm_work(precision, basis, points, cells):
    """(bytes, flops) of a step: the point state read and written once, mass
    and volume read, the node sums and results written and read once."""
    if precision == "fp64":
        per_point, per_node = 2 * (16 + 16 + 32 + 8) + 24, 2 * 56
    else:
        per_point, per_node = 2 * (16 + 8 + 16 + 1) + 8, 36
        if basis == "ugimp":
            per_point += 4
    flops = 350 if basis == "linear" else 700
    return points * per_point + cells * per_node, points * flops


def _dem_work(precision, n, contacts):
    wide = precision == "fp64"
    return (n * (128 if wide else 88) + contacts * (40 if wide else 24),
            n * 40 + contacts * 130)


def work(case):
    k, s = case["kind"], case["steps"]
    if k in ("mpm", "roundtrip"):
        cells, points = case["wc"] * case["hc"], 4 * case["wc"] * case["hc"]
        b, f = _mpm_work(case["precision"], case["basis"], points, cells)
        if k == "roundtrip":  # the host arrays, in and out, every step
            b += points * (88 + 72)
            return dict(bytes=b * s, flops=f * s)
        return dict(bytes=b * s + points * 72, flops=f * s)
    if k == "dem":
        contacts = int((2.8 if case["pitch"] < 2.0e-3 else 0.05) * case["n"])
        b, f = _dem_work(case["precision"], case["n"], contacts)
        return dict(bytes=b * s + case["n"] * 48, flops=f * s)
    if k == "hybrid":
        cells, points = case["wc"] * case["hc"], 4 * case["wc"] * case["hc"]
        b, f = _mpm_work(case["precision"], "ugimp", points, cells)
        db, df = _dem_work(case["precision"], case["n"], 2 * case["n"])
        # coupling: per grain 32 B, per coupled node 24 B (about the grains'
        # cells); the homogenised fields once per step on their nodes
        nodes = (4 * case["wc"] + 5) * (2 * case["hc"] + 9)
        b += db + case["n"] * (32 + 24 + 48)
        return dict(bytes=b * s + points * 72 + case["n"] * 48 + nodes * 48,
                    flops=(f + df + case["n"] * 300) * s)
    bytes_, flops = 0, 0
    for c in _batch_cases(case):
        points = 4 * c["wc"] * c["hc"]
        b, f = _mpm_work("mixed", "linear", points, c["wc"] * c["hc"])
        bytes_, flops = bytes_ + b * s + points * 32, flops + f * s
    return dict(bytes=bytes_, flops=flops)


# ---- 64 bits, plain torch ---------------------------------------------------

def _t(a):
    return torch.as_tensor(a, device="cuda" if torch.cuda.is_available() else "cpu")


class _Axis:
    """Nodes of a basis around positions x along one axis: indices, weights
    and weight derivatives, (points, nodes)."""

    def __init__(self, basis, x, hl, g, h):
        c = torch.floor((x - g) / h).to(torch.int64)
        if basis == "linear":
            self.i = c[:, None] + torch.arange(2, device=x.device)
            d = (x[:, None] - h * self.i.to(x.dtype) - g) / h
            self.w = torch.clamp(1.0 - d.abs(), min=0.0)
            self.g = torch.where(d >= 0.0, -1.0, 1.0).to(x.dtype) / h
            return
        self.i = c[:, None] + torch.arange(-1, 3, device=x.device)
        s = x[:, None] - (h * self.i.to(x.dtype) + g)
        d, l = s.abs(), hl[:, None]
        sg = torch.where(s >= 0.0, -1.0, 1.0).to(x.dtype)
        edge, mid, out = d >= h - l, d >= l, d >= h + l
        w = torch.where(edge, (h + l - d) ** 2 / (2.0 * h),
                        torch.where(mid, 2.0 * l * (1.0 - d / h), 2.0 * l - (l * l + d * d) / h))
        gr = torch.where(edge, sg * (h + l - d) / h,
                         torch.where(mid, sg * 2.0 * l / h, -2.0 * s / h))
        self.w = torch.where(out, torch.zeros_like(w), w) / (2.0 * l)
        self.g = torch.where(out, torch.zeros_like(w), gr) / (2.0 * l)


class _Points64:
    def __init__(self, col):
        p = col["pts"]
        self.q, self.v, self.be = _t(p["q"]).clone(), _t(p["v"]).clone(), _t(p["be"]).clone()
        self.J, self.m, self.vol, self.hl = _t(p["J"]).clone(), _t(p["m"]), _t(p["vol"]), _t(p["hl"])
        self.basis, self.h, self.planes, self.alpha = col["basis"], col["h"], col["planes"], col["alpha"]
        # whole cells about the centre of the asked-for extent
        ends = list(zip(col["gmin"], col["gmax"]))
        self.nx, self.ny = (math.ceil((b - a) / self.h) for a, b in ends)
        self.gmin = tuple(0.5 * (a + b) - 0.5 * (k * self.h)
                          for (a, b), k in zip(ends, (self.nx, self.ny)))
        self.nn = (self.nx + 1) * (self.ny + 1)
        k = torch.arange(self.nn, device=self.q.device)
        self.node = torch.stack([self.gmin[0] + self.h * (k % (self.nx + 1)).to(self.q.dtype),
                                 self.gmin[1] + self.h * (k // (self.nx + 1)).to(self.q.dtype)], dim=1)

    def stencil(self, q, hl):
        """(node indices, weights, x and y weight gradients), (points, nodes)."""
        X = _Axis(self.basis, q[:, 0], hl, self.gmin[0], self.h)
        Y = _Axis(self.basis, q[:, 1], hl, self.gmin[1], self.h)
        pair = lambda a, b: (b[:, :, None] * a[:, None, :]).reshape(len(q), -1)  # noqa: E731
        ix, iy = X.i.clamp(0, self.nx), Y.i.clamp(0, self.ny)
        n = (iy[:, :, None] * (self.nx + 1) + ix[:, None, :]).reshape(len(q), -1)
        return n, pair(X.w, Y.w), pair(X.g, Y.w), pair(X.w, Y.g)

    def scatter(self, n, values):
        out = torch.zeros(self.nn, dtype=values.dtype, device=values.device)
        return out.index_add_(0, n.reshape(-1), values.reshape(-1))

    def to_grid(self):
        n, w, gx, gy = self.st = self.stencil(self.q, self.hl)
        J = self.J
        b00, b01, b11 = self.be[:, 0], 0.5 * (self.be[:, 1] + self.be[:, 2]), self.be[:, 3]
        root = torch.sqrt(b00 * b11 - b01 * b01)
        vol, dev = 0.5 * BULK * (J * J - 1.0), 0.5 * SHEAR * (b00 - b11) / root
        off = SHEAR * b01 / root
        on = (J <= 1.0).to(J.dtype) * -self.vol
        s00, s01, s11 = (on * (vol + dev))[:, None], (on * off)[:, None], (on * (vol - dev))[:, None]
        some = (w != 0.0).to(w.dtype)
        self.gm = self.scatter(n, w * self.m[:, None])
        self.gp = torch.stack([self.scatter(n, w * (self.m * self.v[:, c])[:, None])
                               for c in (0, 1)], dim=1)
        self.gf = torch.stack([self.scatter(n, some * (s00 * gx + s01 * gy)),
                               self.scatter(n, some * (s01 * gx + s11 * gy))], dim=1)

    def update_grid(self, dt):
        m = self.gm[:, None]
        f = self.gf + m * torch.tensor(GRAVITY, dtype=m.dtype, device=m.device)
        new = torch.where(m > 0.0, self.gp + dt * f, torch.zeros_like(f))
        for x, nn in self.planes:
            d = nn[0] * (self.node[:, 0] - x[0]) + nn[1] * (self.node[:, 1] - x[1])
            new = torch.where((d > 0.0)[:, None], new, torch.zeros_like(new))
        self.gnew = new

    def to_points(self, dt):
        m = self.gm[:, None]
        has, safe = m > 0.0, torch.where(m > 0.0, m, torch.ones_like(m))
        gv = torch.where(has, self.gnew / safe, torch.zeros_like(self.gnew))
        ga = torch.where(has, (self.gnew - self.gp) / (dt * safe), torch.zeros_like(self.gnew))
        n, w, gx, gy = self.st
        nv, na = gv[n], ga[n]
        Lx = (nv * gx[..., None]).sum(1)
        Ly = (nv * gy[..., None]).sum(1)
        vp, ap = (nv * w[..., None]).sum(1), (na * w[..., None]).sum(1)
        L = torch.stack([Lx, Ly], dim=2)
        b = self.be[:, [0, 2, 1, 3]].reshape(-1, 2, 2) * self.J[:, None, None]
        Lb = L @ b
        b = b + dt * (Lb + Lb.transpose(1, 2))
        det = b[:, 0, 0] * b[:, 1, 1] - b[:, 0, 1] * b[:, 1, 0]
        J = torch.sqrt(det)
        ys = torch.clamp(0.5 * self.alpha * BULK * (1.0 + J) * (1.0 - J), min=0.0)
        eye = torch.eye(2, dtype=b.dtype, device=b.device)
        dev = b - 0.5 * (b[:, 0, 0] + b[:, 1, 1])[:, None, None] * eye
        size = SHEAR * torch.sqrt((dev * dev).sum((1, 2))) / J
        l2 = torch.where(size > ys, ys / torch.where(size > 0.0, size, torch.ones_like(size)),
                         torch.ones_like(ys))
        ddet = dev[:, 0, 0] * dev[:, 1, 1] - dev[:, 0, 1] * dev[:, 1, 0]
        l1 = torch.sqrt(det - l2 * l2 * ddet)
        b = torch.where((size > ys)[:, None, None], l1[:, None, None] * eye + l2[:, None, None] * dev, b)
        J = torch.sqrt(b[:, 0, 0] * b[:, 1, 1] - b[:, 0, 1] * b[:, 1, 0])
        self.J = J
        self.be = (b / J[:, None, None]).reshape(-1, 4)[:, [0, 2, 1, 3]]
        self.v = (1.0 - FLIP) * vp + FLIP * (self.v + dt * ap)
        self.q = self.q + dt * vp
        for x, nn in self.planes:
            d = nn[0] * (self.q[:, 0] - x[0]) + nn[1] * (self.q[:, 1] - x[1])
            hit = (d <= 0.0)[:, None]
            nv = torch.tensor(nn, dtype=d.dtype, device=d.device)
            self.q = torch.where(hit, self.q - d[:, None] * nv, self.q)
            self.v = torch.where(hit, torch.zeros_like(self.v), self.v)

    def step(self, dt):
        self.to_grid()
        self.update_grid(dt)
        self.to_points(dt)

    def outputs(self):
        return {k: getattr(self, k).cpu().numpy() for k in ("q", "v", "be", "J")}


def _cross(a, b):
    return a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]


def _perp(a):
    return torch.stack([-a[:, 1], a[:, 0]], dim=1)


def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _norm(a):
    return torch.sqrt(_dot(a, a))


class _Disks64:
    """Candidate pairs are listed once, 1 mm beyond contact; ``far`` says when
    the disks have moved too far for the list."""

    SKIN = 1.0e-3

    def __init__(self, sc):
        self.q, self.v = _t(sc["q"]).clone(), _t(sc["v"]).clone()
        self.r, self.m, self.I = _t(sc["r"]), _t(sc["m"]), _t(sc["I"])
        self.fixed, self.planes = _t(sc["fixed"]) != 0, sc["planes"]
        self.q0 = self.q.clone()
        self.list_pairs()
        k = len(self.r) * len(self.planes)
        dev = self.q.device
        self.ds = torch.zeros(len(self.a) + k, 2, dtype=torch.float64, device=dev)
        self.pa = torch.arange(len(self.r), device=dev).repeat(len(self.planes))
        self.px = torch.cat([torch.tensor(x, dtype=torch.float64, device=dev).expand(len(self.r), 2)
                             for x, _ in self.planes])
        self.pn = torch.cat([torch.tensor(n, dtype=torch.float64, device=dev).expand(len(self.r), 2)
                             for _, n in self.planes])

    def list_pairs(self):
        x, n = self.q[:, :2], len(self.r)
        H = 2.0 * float(self.r.max()) + self.SKIN
        c = torch.floor((x - x.min(0).values) / H).to(torch.int64) + 1
        row = int(c[:, 0].max()) + 3
        key = c[:, 1] * row + c[:, 0]
        skey, order = torch.sort(key, stable=True)
        A, B = [], []
        for off in (0, 1, row - 1, row, row + 1):
            lo = torch.searchsorted(skey, key + off)
            cnt = torch.searchsorted(skey, key + off, right=True) - lo
            a = torch.repeat_interleave(torch.arange(n, device=x.device), cnt)
            start = torch.cumsum(cnt, 0) - cnt
            b = order[lo[a] + torch.arange(len(a), device=x.device) - start[a]]
            keep = (a < b) if off == 0 else (a != b)
            a, b = torch.minimum(a, b)[keep], torch.maximum(a, b)[keep]
            d = x[a] - x[b]
            keep = (d * d).sum(1) <= (self.r[a] + self.r[b] + self.SKIN) ** 2
            A.append(a[keep])
            B.append(b[keep])
        a, b = torch.cat(A), torch.cat(B)
        # a fixed disk is the second of its pair; two fixed ones are no pair
        swap = self.fixed[a]
        a, b = torch.where(swap, b, a), torch.where(swap, a, b)
        keep = ~(self.fixed[a] & self.fixed[b])
        self.a, self.b = a[keep], b[keep]
        self.kin = self.fixed[self.b]

    def far(self):
        d = self.q[:, :2] - self.q0[:, :2]
        return float((d * d).sum(1).max()) > (0.5 * self.SKIN) ** 2

    def law(self, act, n, depth, vrel, dt):
        """Forces of the contacts in act (indices into ds); every other
        contact's spring is dropped."""
        kn, kt, gn, gt, mu = _penalty()
        ds = self.ds[act] + dt * vrel
        ds = ds - _dot(n, ds) * n
        vt = vrel - _dot(n, vrel) * n
        fn = -kn * depth * n - 0.5 * gn * (vrel - vt)
        ft = -kt * ds - 0.5 * gt * vt
        cap = mu * _norm(fn)
        vn = _norm(vt)
        slip = 0.5 * gt * vn > cap
        slide = ~slip & (_norm(ft) > cap)
        A = kt * kt * _dot(ds, ds)
        B = kt * gt * _dot(ds, vt)
        C = 0.25 * gt * gt * _dot(vt, vt) - mu * mu * _dot(fn, fn)
        root = torch.sqrt(torch.clamp(B * B - 4.0 * A * C, min=0.0))
        lam = torch.where(B > 0.0, (2.0 * C) / (-B - root), (-B + root) / (2.0 * A))
        nds = torch.where(slide, lam * ds, ds)
        ft = torch.where(slide, -kt * nds - 0.5 * gt * vt, ft)
        ft = torch.where(slip, -cap * vt / torch.where(vn > 0.0, vn, torch.ones_like(vn)), ft)
        self.ds = torch.zeros_like(self.ds)
        self.ds[act] = torch.where(slip, torch.zeros_like(nds), nds)
        return fn + ft

    def step(self, dt):
        x, v, w, r = self.q[:, :2], self.v[:, :2], self.v[:, 2:], self.r
        a, b = self.a, self.b
        d = x[a] - x[b]
        hit = torch.nonzero((d * d).sum(1) - (r[a] + r[b]) ** 2 <= 0.0)[:, 0]
        a, b, d, kin = a[hit], b[hit], d[hit], self.kin[hit][:, None]
        dist = _norm(d)
        n = d / dist
        ra, rb = r[a][:, None], r[b][:, None]
        r0 = torch.where(kin, -ra * n, -d * (ra / (ra + rb)))
        r1 = d + r0
        vrel = (v[a] + w[a] * _perp(r0)) - (v[b] + w[b] * _perp(r1))
        depth = torch.clamp(dist - ra - rb, max=0.0)
        gap = _dot(self.pn, x[self.pa] - self.px)[:, 0] - r[self.pa]
        pl = torch.nonzero((gap <= 0.0) & ~self.fixed[self.pa])[:, 0]
        pa, pn = self.pa[pl], self.pn[pl]
        p0 = -r[pa][:, None] * pn
        pv = v[pa] + w[pa] * _perp(p0)
        f = self.law(torch.cat([hit, len(self.a) + pl]), torch.cat([n, pn]),
                     torch.cat([depth, gap[pl][:, None]]), torch.cat([vrel, pv]), dt)
        fc, fp = f[: len(hit)], f[len(hit):]
        F = self.m[:, None] * torch.tensor(GRAVITY, dtype=f.dtype, device=f.device)
        T = torch.zeros_like(self.I)
        F.index_add_(0, pa, fp)
        T.index_add_(0, pa, _cross(p0, fp))
        F.index_add_(0, a, fc)
        T.index_add_(0, a, _cross(r0, fc))
        free = ~kin[:, 0]
        F.index_add_(0, b[free], -fc[free])
        T.index_add_(0, b[free], -_cross(r1[free], fc[free]))
        F[self.fixed], T[self.fixed] = 0.0, 0.0
        # circle-circle contacts, for the homogenised stress
        self.cc = (a[free], b[free], (x[a] + r0)[free], fc[free])
        self.v = self.v + dt * torch.cat([F / self.m[:, None], (T / self.I)[:, None]], dim=1)
        self.q = self.q + dt * self.v

    def outputs(self):
        return dict(q=self.q.cpu().numpy(), v=self.v.cpu().numpy())


def _exact_hybrid(case, seed):
    col, sc = _hybrid_scene(case, seed)
    P, D, dt, h = _Points64(col), _Disks64(sc), col["dt"], col["h"]
    stress, velocity = _t(np.zeros((P.nn, 4))), _t(np.zeros((P.nn, 2)))
    ext = P.hl[0].expand(len(D.r))

    def span(x, ax):  # inclusive node range of a grain's extent
        g = P.gmin[ax]
        return (torch.floor((x - P.hl[0] - g) / h).to(torch.int64),
                torch.ceil((x + P.hl[0] - g) / h).to(torch.int64))

    for _ in range(case["steps"]):
        before = D.q.clone()
        P.to_grid()
        (x0, x1), (y0, y1) = span(before[:, 0], 0), span(before[:, 1], 1)
        coupled = ~D.fixed
        for ky in range(4):
            for kx in range(4):
                ix, iy = x0 + kx, y0 + ky
                inside = (ix <= x1) & (iy <= y1) & (ix >= 0) & (iy >= 0) & (ix <= P.nx) & (iy <= P.ny)
                node = iy.clamp(0, P.ny) * (P.nx + 1) + ix.clamp(0, P.nx)
                coupled = coupled & ~(inside & (P.gm[node] <= 1.0e-6))
        c = torch.nonzero(coupled)[:, 0]
        n, w, _, _ = P.stencil(before[c, :2], ext[c])
        gm = P.scatter(n, w * D.m[c][:, None])[:, None]
        D.step(dt)
        P.update_grid(dt)
        gp = torch.stack([P.scatter(n, w * (D.m[c] * D.v[c, k])[:, None]) for k in (0, 1)], dim=1)
        on, m = gm > 0.0, P.gm[:, None]
        lam = torch.where(on, (gm * P.gnew - m * gp) / torch.where(on, m + gm, torch.ones_like(m)),
                          torch.zeros_like(gp))
        P.gnew = P.gnew - lam
        acc = lam / torch.where(on, gm, torch.ones_like(gm))
        vel = D.v[c, :2] + (acc[n] * w[..., None]).sum(1)
        D.v[c, :2] = vel
        D.q[c, :2] = before[c, :2] + dt * vel
        P.to_points(dt)
        a, b, at, f = D.cc
        rel = D.q[a, :2] - D.q[b, :2]
        quarter = torch.full_like(D.r, 0.25 * h)
        n, w, _, _ = P.stencil(at, quarter[: len(at)] if len(at) <= len(D.r)
                               else torch.full_like(at[:, 0], 0.25 * h))
        s00, s11 = -f[:, 0] * rel[:, 0], -f[:, 1] * rel[:, 1]
        s01 = -0.5 * (f[:, 0] * rel[:, 1] + f[:, 1] * rel[:, 0])
        for k, s in enumerate((s00, s01, s01, s11)):
            stress[:, k] += P.scatter(n, w * (s / (h * h))[:, None])
        free = torch.nonzero(~D.fixed)[:, 0]
        n, w, _, _ = P.stencil(D.q[free, :2], quarter[free])
        mass = P.scatter(n, w * D.m[free][:, None])
        for k in (0, 1):
            mom = P.scatter(n, w * (D.m[free] * D.v[free, k])[:, None])
            velocity[:, k] += torch.where(mass > 0.0, mom / torch.where(mass > 0.0, mass, torch.ones_like(mass)),
                                          torch.zeros_like(mom))
    if D.far():
        return None
    return dict(points=P.outputs(), grains=D.outputs(), stress=stress.cpu().numpy(),
                velocity=velocity.cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mpm", "roundtrip"):
        col = _column(case, seed)
        P = _Points64(col)
        for _ in range(case["steps"]):
            P.step(col["dt"])
        return P.outputs()
    if kind == "dem":
        D = _Disks64(_disks(case, seed))
        for _ in range(case["steps"]):
            D.step(case["dt"])
        return None if D.far() else D.outputs()
    if kind == "hybrid":
        return _exact_hybrid(case, seed)
    if case["members"] * case["steps"] * 2.5e-3 > EXACT_SECONDS:
        return None
    got = []
    for i, c in enumerate(_batch_cases(case)):
        col = _column(c, int(seed) + 1000 * i)
        P = _Points64(col)
        for _ in range(case["steps"]):
            P.step(col["dt"])
        got.append(P.outputs())
    return dict(q=np.concatenate([g["q"] for g in got]), v=np.concatenate([g["v"] for g in got]))

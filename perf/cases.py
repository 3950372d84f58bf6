"""The workloads whose time is followed: what a user of the package has it do.

Every case goes through the public entry points of ``newrecon_gb300``:

* the OSTR loop over a resident scan (``OSTR.iterate``) and the whole call
  (``reconstruct``) at the package's own workloads (tiny, small, clinical,
  full resolution) and at the scanner geometry that the module-level defaults
  of ``newrecon_gb300.ostr`` describe (several views per subset, scatter);
* a batch of uneven cases (``Batch``), the OS-SART loop (``OSSART``), the
  reference-shaped calls one by one (``fprojectCB_1R_GPU_OSTR_cos`` ...), the
  FP64 objective, the dual-energy subtraction;
* the warm-start network, forward on a volume and loss + gradients on a batch
  of training patches.

Scans are synthetic and seeded: ellipsoids in a breast-shaped body, projected
analytically here (not by the package), with Poisson counts.  ``exact`` is the
same mathematics in 64 bits in plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from newrecon_gb300 import dual_energy, ostr, sart, warmstart
from newrecon_gb300.geometry import Geometry, view_angles

MU_BODY, MU_GLAND, MU_CALC = 0.0456, 0.0802, 2.0  # 1/mm, as the package's phantoms
WARMSTART_PARAMS = "newrecon_gb300/data/warmstart_clinical.npz"
WEIGHTS = list(dual_energy.DEFAULT_WEIGHTS)


# ---------------------------------------------------------------------------
# The cases.

def _scan(kind, nx, ny, nz, vxy, nbx, nby, bin_size, views, span, subsets, iters, potential,
          beta, delta, I0, **more):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, vxy=vxy, nbx=nbx, nby=nby, bin=bin_size,
             views=views, span=span, subsets=subsets, iters=iters, potential=potential,
             beta=beta, delta=delta, I0=I0, scatter=False, scanner=False)
    c.update(more)
    return c


def listed():
    return [
        # the smallest whole call: a test-sized volume, host arrays in, volume out
        dict(_scan("recon", 40, 24, 8, 0.8, 48, 32, 0.8, 6, 15.0, 3, 2, "lange", 20.0, 0.01, 1e4),
             name="recon_tiny"),
        # a low-resolution preview from host arrays: the whole call, 10 iterations
        dict(_scan("recon", 256, 128, 24, 0.4, 320, 160, 0.4, 9, 12.0, 9, 10, "hyperbola", 50.0,
                   0.002, 1e4), name="recon_small"),
        # the clinical workload: one of the 50 iterations, scan resident
        dict(_scan("iterate", 1024, 512, 60, 0.14, 1664, 832, 0.14, 25, 25.0, 25, 1, "huber",
                   100.0, 0.003, 5e3), name="iterate_clinical"),
        # the full-resolution workload: one iteration
        dict(_scan("iterate", 2048, 1024, 70, 0.085, 3328, 1664, 0.085, 15, 7.5, 15, 1,
                   "hyperbola", 200.0, 0.002, 4e3), name="iterate_fullres"),
        # the scanner that the module-level defaults describe: five views per
        # subset, the Lange prior, measured scatter; set-up and one iteration
        dict(_scan("recon", 2000, 1000, 48, 0.085, 3584, 1400, 0.085, 25, 25.0, 5, 1, "lange",
                   150000.0, 0.003, 5e3, scatter=True, scanner=True), name="recon_scanner"),
        # a queue of uneven cases (in-plane size, thickness, views) advanced together
        dict(kind="batch", n=4, scale=0.75, iters=1, name="batch_mixed"),
        # OS-SART with the hyperbola prior on the clinical scan, one iteration
        dict(_scan("ossart", 1024, 512, 60, 0.14, 1664, 832, 0.14, 25, 25.0, 25, 1, "hyperbola",
                   -0.2, 0.003, 5e3, cos=True, regularized=True, supersample=False),
             name="ossart_clinical"),
        # a script on the reference-shaped calls: one subset of views, odd sizes
        dict(_scan("calls", 701, 353, 45, 0.2, 835, 421, 0.2, 15, 15.0, 3, 1, "lange", 150.0,
                   0.003, 1e4), name="calls_odd"),
        # the FP64 objective that monotone runs check
        dict(_scan("objective", 1024, 512, 60, 0.14, 1664, 832, 0.14, 25, 25.0, 25, 1, "huber",
                   100.0, 0.003, 5e3), name="objective_clinical"),
        # the dual-energy sweep over two reconstructions, nine weights
        dict(kind="dual", nx=1024, ny=512, nz=60, weights=9, mask=False, name="dual_clinical"),
        # the warm-start network on a clinical volume
        dict(kind="cnn_forward", nx=1024, ny=512, nz=60, nb=1, name="cnn_forward_clinical"),
        # its loss and gradients on the default training batch of patches
        dict(kind="cnn_grad", nx=126, ny=32, nz=16, nb=8, name="cnn_grad_patches"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "recon", "batch", "ossart", "calls", "objective",
                       "dual", "cnn_forward", "cnn_grad"])
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(2, 6), scale=round(_log(rng, 0.15, 0.75), 3), iters=1)
    if kind == "dual":
        return dict(kind=kind, nx=int(_log(rng, 40, 1024)), ny=int(_log(rng, 24, 512)),
                    nz=rng.randint(8, 60), weights=rng.randint(1, 9), mask=rng.random() < 0.5)
    if kind == "cnn_forward":
        return dict(kind=kind, nx=int(_log(rng, 96, 1024)), ny=int(_log(rng, 32, 512)),
                    nz=rng.randint(12, 60), nb=1)
    if kind == "cnn_grad":
        return dict(kind=kind, nx=rng.choice([96, 126, 128, 140]), ny=rng.randint(16, 32),
                    nz=rng.randint(8, 16), nb=rng.randint(2, 8))
    top = {"calls": 700, "recon": 1024}.get(kind, 1536)
    nx = int(_log(rng, 40, top))
    ny = max(16, int(nx * rng.uniform(0.4, 0.6)))
    nz = rng.randint(8, 64)
    vxy = 0.085 if nx > 1200 else round(rng.uniform(0.85, 1.1) * 150.0 / max(nx, 375), 3)
    views, subsets = rng.choice([(9, 9), (15, 15), (15, 5), (25, 25), (25, 5), (24, 12)])
    c = _scan(kind, nx, ny, nz, vxy, int(nx * rng.uniform(1.1, 1.6)), int(ny * rng.uniform(1.1, 1.6)),
              vxy, views, round(rng.uniform(7.5, 25.0), 2), subsets, 1,
              rng.choice(["q2", "lange", "hyperbola", "huber"]), round(_log(rng, 20, 500), 1),
              rng.choice([0.002, 0.003, 0.01]), round(_log(rng, 3e3, 2e4)))
    if kind in ("iterate", "recon"):
        c["scatter"] = rng.random() < 0.4
        c["iters"] = 1 if nx > 500 else rng.randint(1, 3)
    if kind == "ossart":
        c.update(beta=-0.2, cos=rng.random() < 0.5, regularized=rng.random() < 0.5,
                 supersample=rng.random() < 0.3)
    if kind == "calls" and c["potential"] not in ("q2", "lange"):
        c["potential"] = "lange"  # the two priors that have a call of their own
    return c


# ---------------------------------------------------------------------------
# Inputs.

def _geometry(c):
    if c["scanner"]:
        # the module-level defaults of newrecon_gb300.ostr
        return Geometry(nx=c["nx"], ny=c["ny"], nz=c["nz"], vx=c["vxy"], vy=c["vxy"], vz=1.0,
                        x_p0=-93.5, y_p0=-85.0, z_p0=-30.0, nbx=c["nbx"], nby=c["nby"],
                        bx=c["bin"], by=c["bin"], x_d0=-152.32, y_d0=-119.0, detectorR=47.0,
                        sourceR=608.5, sourceY=0.0, n_angles=c["views"])
    return Geometry.dbt(c["nx"], c["ny"], c["nz"], c["vxy"], 1.0, c["nbx"], c["nby"], c["bin"],
                        c["views"])


class _Geo:
    """The geometry as the package is given it (float32 fields), in 64 bits."""

    def __init__(self, g):
        for f in ("vx", "vy", "vz", "x_p0", "y_p0", "z_p0", "bx", "by", "x_d0", "y_d0",
                  "detectorR", "sourceR", "sourceY"):
            setattr(self, f, float(np.float32(getattr(g, f))))
        for f in ("nx", "ny", "nz", "nbx", "nby"):
            setattr(self, f, int(getattr(g, f)))

    def source(self, theta):
        t = float(theta)
        return self.sourceR * math.sin(t), self.sourceY, self.sourceR * math.cos(t)

    def bins(self, sub=1):
        """Bin (or sub-bin) centres along i and j, float64 on the device."""
        i = torch.arange(self.nbx * sub, dtype=torch.float64, device="cuda")
        j = torch.arange(self.nby * sub, dtype=torch.float64, device="cuda")
        return (self.x_d0 + (i + 0.5) * self.bx / sub, self.y_d0 + (j + 0.5) * self.by / sub)


def _ellipsoids(g, seed):
    """(centre, semi-axes, added attenuation) of the body and what lies in it."""
    rng = np.random.default_rng([seed, 17])
    wx, wy, wz = g.nx * g.vx, g.ny * g.vy, g.nz * g.vz
    cx, cy, cz = g.x_p0 + wx / 2, g.y_p0 + wy, g.z_p0 + wz / 2
    body = (np.array([cx, cy, cz]), np.array([0.45 * wx, 0.85 * wy, 0.8 * wz]), MU_BODY)
    out = [body]
    for _ in range(20):
        u = rng.uniform([-0.7, -0.9, -0.5], [0.7, -0.05, 0.5])
        s = rng.uniform(0.03, 0.12, size=3) * np.array([wx, wy, wz * 2.0])
        out.append((body[0] + u * body[1] * 0.75, s, MU_GLAND - MU_BODY))
    for _ in range(4):
        u = rng.uniform([-0.5, -0.7, -0.4], [0.5, -0.1, 0.4])
        out.append((body[0] + u * body[1], np.full(3, rng.uniform(0.25, 0.5)), MU_CALC - MU_BODY))
    return out


def _lines(g, angles, ells):
    """Line integrals [view][i][j] of the ellipsoids (float32, analytic)."""
    G = _Geo(g)
    bx, by = (v.float() for v in G.bins())
    out = torch.empty(len(angles), G.nbx, G.nby, device="cuda")
    for a, th in enumerate(angles):
        s = G.source(th)
        dx, dy, dz = (bx - s[0])[:, None], (by - s[1])[None, :], -G.detectorR - s[2]
        L = torch.sqrt(dx * dx + dy * dy + dz * dz)
        tot = torch.zeros(G.nbx, G.nby, device="cuda")
        for c, r, mu in ells:
            o = [(s[k] - float(c[k])) / float(r[k]) for k in range(3)]
            ex, ey, ez = dx / float(r[0]), dy / float(r[1]), dz / float(r[2])
            A = ex * ex + ey * ey + ez * ez
            B = ex * o[0] + ey * o[1] + ez * o[2]
            D = B * B - A * (o[0] ** 2 + o[1] ** 2 + o[2] ** 2 - 1.0)
            tot += mu * 2.0 * torch.sqrt(D.clamp_min(0.0)) / A * L
        out[a] = tot.clamp_min(0.0)
    return out


def _volume(g, seed, ells):
    """A plausible iterate [z][y][x]: the ellipsoids on the grid, damped, with noise."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 7 + 3)
    ax = [torch.arange(n, device="cuda") * v + (p + v / 2)
          for n, v, p in ((g.nx, g.vx, g.x_p0), (g.ny, g.vy, g.y_p0), (g.nz, g.vz, g.z_p0))]
    vol = torch.zeros(g.nz, g.ny, g.nx, device="cuda")
    for c, r, mu in ells:
        q = [((ax[k] - float(c[k])) / float(r[k])) ** 2 for k in range(3)]
        lo, hi = [], []
        for k in range(3):
            on = torch.nonzero(q[k] <= 1.0)
            lo.append(int(on[0]) if len(on) else 0)
            hi.append(int(on[-1]) + 1 if len(on) else 0)
        sub = vol[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]
        sub += 0.9 * mu * (q[2][lo[2]:hi[2], None, None] + q[1][None, lo[1]:hi[1], None]
                           + q[0][None, None, lo[0]:hi[0]] <= 1.0)
    noise = torch.randn(vol.shape, device="cuda", generator=gen)
    vol += 0.004 * noise * (vol > 0) + 0.001 * noise.abs_() * (vol <= 0)
    return vol.clamp_(min=0.0).view(-1)


def _inputs(c, seed):
    g = _geometry(c)
    angles = view_angles(c["views"], c["span"])
    ells = _ellipsoids(g, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed * 11 + 5)
    line = _lines(g, angles, ells)
    b = torch.full_like(line, float(c["I0"]))
    mean = b * torch.exp(-line)
    r = None
    if c["scatter"]:
        r = torch.full_like(line, 0.05 * float(c["I0"])) * (0.5 + 0.5 * torch.exp(-line))
        mean = mean + r
    y = torch.poisson(mean, generator=gen)
    return dict(g=g, angles=angles, ells=ells, y=y.view(-1), b=b.view(-1),
                r=None if r is None else r.reshape(-1), x0=_volume(g, seed, ells))


def _order(views, subsets):
    """Subset-major view order: position i * Vs + j holds view j * M + i."""
    vs = views // subsets
    return np.array([(p % vs) * subsets + p // vs for p in range(views)], np.int32)


def _batch_cases(c, seed):
    """Uneven cases with the spread of the package's batched workload."""
    rng = np.random.default_rng(99)  # the sizes belong to the case, not to the seed
    out = []
    for k in range(c["n"]):
        views = [15, 9, 25, 15, 9, 25][k]
        pot = ["hyperbola", "hyperbola", "huber", "hyperbola", "lange", "hyperbola"][k]
        s = c["scale"]
        out.append(_scan("iterate", int(rng.uniform(512, 1024) * s), int(rng.uniform(256, 512) * s),
                         int(rng.uniform(30, 80) * s), round(0.14 / s, 4), int(1664 * s),
                         int(832 * s), round(0.14 / s, 4), views,
                         float(round(rng.uniform(7.5, 25.0), 2)), views, c["iters"], pot, 50.0,
                         0.002, 1e4))
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        cases, x0 = [], []
        for k, s in enumerate(_batch_cases(c, seed)):
            i = _inputs(s, seed * 10 + k)
            cases.append(dict(geom=i["g"], angles=i["angles"], prj=i["y"], blank=i["b"],
                              subset_num=s["subsets"], iter_num=s["iters"], beta=s["beta"],
                              delta=s["delta"], potential=s["potential"], x0=i["x0"]))
            x0.append(i["x0"])
        return dict(kind=kind, batch=ostr.Batch(cases), x0=x0)
    if kind == "dual":
        g = Geometry.dbt(c["nx"], c["ny"], c["nz"], 0.14, 1.0, 8, 8, 0.14, 1)
        e = _ellipsoids(g, seed)
        he = _volume(g, seed, e)
        le = _volume(g, seed + 1, [(a, b, 1.7 * m) for a, b, m in e])
        return dict(kind=kind, he=he, le=le, w=WEIGHTS[:c["weights"]], shape=(c["nx"], c["ny"]),
                    z=c["nz"] // 2, level=0.03 if c["mask"] else None)
    if kind in ("cnn_forward", "cnn_grad"):
        dims = (c["nx"], c["ny"], c["nz"], c["nb"])
        g = Geometry.dbt(c["nx"], c["ny"], c["nz"] * c["nb"], 0.14, 1.0, 8, 8, 0.14, 1)
        x = _volume(g, seed, _ellipsoids(g, seed))
        net = warmstart.load(WARMSTART_PARAMS)
        if kind == "cnn_forward":
            return dict(kind=kind, net=net, x=x, dims=dims)
        gen = torch.Generator(device="cuda").manual_seed(seed + 23)
        t = x + 0.003 * torch.randn(x.shape, device="cuda", generator=gen)
        return dict(kind=kind, net=net, x=x, t=t, dims=dims)
    i = _inputs(c, seed)
    if kind == "recon":
        host = [None if t is None else t.cpu().numpy() for t in (i["y"], i["b"], i["r"])]
        if c["scanner"]:  # scans of this size stay on the card between calls
            host = [i["y"], i["b"], i["r"]]
        return dict(kind=kind, c=c, g=i["g"], angles=i["angles"], scan=host)
    if kind == "ossart":
        line = torch.log(i["b"] / i["y"].clamp_min(1.0))
        plan = sart.OSSART(i["g"], subset_num=c["subsets"], lam=0.8, use_cos=c["cos"],
                           regularized=c["regularized"], beta=c["beta"], delta=c["delta"],
                           supersample=c["supersample"])
        plan.setup(i["angles"], line)
        return dict(kind=kind, plan=plan, x0=i["x0"], iters=c["iters"])
    if kind == "calls":
        idx = _order(c["views"], c["subsets"])
        vs, n = c["views"] // c["subsets"], i["g"].n_bins
        first = vs  # the second subset
        pick = torch.from_numpy(idx[first:2 * vs].astype(np.int64)).cuda()
        d = float(c["I0"]) * 600.0 * 0.3 * c["views"] * (0.5 + i["x0"])
        return dict(kind=kind, c=c, g=i["g"], x=i["x0"], d=d, a0=first, a1=2 * vs,
                    y=i["y"].view(c["views"], n)[pick].reshape(-1),
                    b=i["b"].view(c["views"], n)[pick].reshape(-1),
                    angles=torch.from_numpy(i["angles"]).cuda(), idx=torch.from_numpy(idx).cuda())
    plan = ostr.OSTR(i["g"], subset_num=c["subsets"], beta=c["beta"], delta=c["delta"],
                     potential=c["potential"], has_scatter=c["scatter"])
    plan.setup(i["angles"], i["y"], i["b"], i["r"])
    return dict(kind=kind, plan=plan, x0=i["x0"], iters=c["iters"])


def run(state):
    kind = state["kind"]
    if kind == "recon":
        c = state["c"]
        y, b, r = state["scan"]
        return ostr.reconstruct(state["g"], y, b, r, angles=state["angles"],
                                subset_num=c["subsets"], iter_num=c["iters"], beta=c["beta"],
                                delta=c["delta"], potential=c["potential"])
    if kind in ("iterate", "ossart"):
        return state["plan"].iterate(state["x0"].clone(), state["iters"])
    if kind == "batch":
        for x, x0 in zip(state["batch"].x, state["x0"]):
            x.copy_(x0)
        return list(state["batch"].run())
    if kind == "calls":
        c, g, x = state["c"], state["g"], state["x"]
        ostr.set_geometry(g)
        ostr.beta = c["beta"]
        args = (state["angles"], state["idx"], state["a0"], state["a1"])
        line = torch.zeros_like(state["y"])
        ostr.fprojectCB_1R_GPU_OSTR_cos(x, line, *args)
        h = ostr.compute_h(state["y"], state["b"], line, None)
        capL = torch.zeros_like(x)
        ostr.bprojectCB_GPU_SBP(capL, h, state["idx"], state["angles"], state["a0"], state["a1"])
        capL = ostr.temp_fun2(c["subsets"], x.numel(), capL)
        RDD, RD = torch.zeros_like(x), torch.zeros_like(x)
        if c["potential"] == "q2":
            ostr.prior_GPU_OSTR_Q2(RDD, RD, x, g.z_xy_ratio)
        else:
            ostr.prior_GPU_OSTR(RDD, RD, x, c["delta"], g.z_xy_ratio)
        return [line, h, capL, RDD, RD, ostr.update_est(x, capL, RD, state["d"], RDD)]
    if kind == "objective":
        return list(state["plan"].objective(state["x0"]))
    if kind == "dual":
        d, ent = dual_energy.subtract(state["he"], state["le"], state["w"],
                                      slice_shape=state["shape"], entropy_slice=state["z"],
                                      mask_level=state["level"])
        return [d] + ent
    if kind == "cnn_forward":
        return state["net"].forward(state["x"], state["dims"])
    loss, grad = state["net"].loss_grad(state["x"], state["t"], state["dims"])
    return [loss, grad]


# ---------------------------------------------------------------------------
# What a pass cannot do without.

def _segments(g, angles):
    """Voxel crossings of all rays that meet the volume (an estimate from the
    mean slopes; 2 operations each)."""
    G = _Geo(g)
    tot = 0.0
    for th in angles:
        sx, _, sz = G.source(th)
        depth = sz + G.detectorR
        mag = depth / max(sz - (G.z_p0 + 0.5 * G.nz * G.vz), 1.0)
        wx, wy = G.nx * G.vx * mag, G.ny * G.vy * mag
        rays = min(wx, G.nbx * G.bx) * min(wy, G.nby * G.by) / (G.bx * G.by)
        slope_x = max(abs(sx) / depth, 0.25 * wx / depth)
        slope_y = 0.5 * wy / depth
        tot += rays * G.nz * (1.0 + slope_x * G.vz / G.vx + slope_y * G.vz / G.vy)
    return tot


def _loop_work(c, updates_read, prior):
    g = _geometry(c)
    n, bins = g.n_voxels, g.n_bins
    seg = _segments(g, view_angles(c["views"], c["span"]))
    sub = c["iters"] * c["subsets"]
    data = 3 if c["scatter"] else 2
    by = sub * 4.0 * n * updates_read + c["iters"] * c["views"] * bins * 4.0 * data
    fl = c["iters"] * (2.0 * seg + c["views"] * n * 20.0) + sub * n * (26.0 * prior + 6.0)
    return by, fl


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        parts = [_loop_work(s, 3, 7.0) for s in _batch_cases(c, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "dual":
        n = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 4.0 * n * (2 + c["weights"]), "flops": 2.0 * n * c["weights"]}
    if kind in ("cnn_forward", "cnn_grad"):
        n = c["nx"] * c["ny"] * c["nz"] * c["nb"]
        fl = n * 2.0 * 27 * (32 + 4 * 32 * 32 + 32)
        if kind == "cnn_forward":
            return {"bytes": 8.0 * n, "flops": fl}
        return {"bytes": 8.0 * n, "flops": 3.0 * fl}
    g = _geometry(c)
    n, bins = g.n_voxels, g.n_bins
    if kind == "ossart":
        # x read, x written per sub-iteration; line integrals and chords per view
        by, fl = _loop_work(dict(c, scatter=False), 2, 7.0 if c["regularized"] else 0.0)
        return {"bytes": by, "flops": fl * (2.0 if c["supersample"] else 1.0)}
    if kind == "calls":
        vs = c["views"] // c["subsets"]
        seg = _segments(g, view_angles(c["views"], c["span"])) / c["subsets"]
        return {"bytes": 4.0 * (7 * n + 4 * vs * bins),
                "flops": 2.0 * seg + n * (20.0 * vs + 26 * 7.0 + 6.0)}
    if kind == "objective":
        seg = _segments(g, view_angles(c["views"], c["span"]))
        return {"bytes": 4.0 * (n + 2 * c["views"] * bins), "flops": 2.0 * seg + n * 13 * 7.0}
    # x read, d read, x written per sub-iteration; counts and blank scan per view
    by, fl = _loop_work(c, 3, 7.0)
    if kind == "recon":  # set-up: every count once more, d written
        by += c["views"] * bins * 4.0 + 4.0 * n
        fl += c["views"] * n * 20.0
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# The same results in 64 bits.

def _project64(G, x, theta, sub=1):
    """(line integral, chord) [i][j] of the rays of one view through x [z][y][x]."""
    s = G.source(theta)
    bx, by = G.bins(sub)
    n = (G.nx, G.ny, G.nz)
    v = (G.vx, G.vy, G.vz)
    p = (G.x_p0, G.y_p0, G.z_p0)
    shape = (bx.numel(), by.numel())
    d = [(bx - s[0])[:, None].expand(shape).reshape(-1), (by - s[1])[None, :].expand(shape).reshape(-1)]
    d.append(torch.full_like(d[0], -G.detectorR - s[2]))
    L = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    lo, hi = None, None
    for k in range(3):
        dk = torch.where(d[k] == 0, torch.full_like(d[k], 1e-30), d[k])
        d[k] = dk
        a0, a1 = (p[k] - s[k]) / dk, (p[k] + n[k] * v[k] - s[k]) / dk
        m, q = torch.minimum(a0, a1), torch.maximum(a0, a1)
        lo = m if lo is None else torch.maximum(lo, m)
        hi = q if hi is None else torch.minimum(hi, q)
    ray = torch.nonzero(lo < hi).view(-1)
    out, chord = torch.zeros_like(L), torch.zeros_like(L)
    if ray.numel() == 0:
        return out.view(shape), chord.view(shape)
    a, end, L = lo[ray], hi[ray], L[ray]
    chord[ray] = (end - a) * L
    stride = (1, n[0], n[0] * n[1])
    cell, nxt, step, move = None, [], [], []
    for k in range(3):
        dk = d[k][ray]
        i = torch.floor((s[k] + a * dk - p[k]) / v[k]).clamp_(0, n[k] - 1)
        cell = i * stride[k] if cell is None else cell + i * stride[k]
        up = dk > 0
        nxt.append((p[k] + (i + up) * v[k] - s[k]) / dk)
        step.append(v[k] / dk.abs())
        move.append(torch.where(up, stride[k], -stride[k]))
    cell = cell.long()
    tot = torch.zeros_like(a)
    last = x.numel() - 1
    while True:
        if not bool((a < end).any()):
            break
        for _ in range(16):
            m = torch.minimum(torch.minimum(nxt[0], nxt[1]), torch.minimum(nxt[2], end))
            tot += (m - a).clamp_(min=0.0) * x[cell.clamp(0, last)]
            a = torch.maximum(a, m)
            for k in range(3):
                hit = nxt[k] <= m
                nxt[k] = torch.where(hit, nxt[k] + step[k], nxt[k])
                cell = torch.where(hit, cell + move[k], cell)
    out[ray] = tot * L
    return out.view(shape), chord.view(shape)


def _taps64(pos, n):
    lb = torch.floor(pos)
    lb = torch.where(pos < lb + 0.5, lb - 1, lb)
    f = pos - (lb + 0.5)
    lb = lb.long()
    return (lb.clamp(0, n - 1), (lb + 1).clamp(0, n - 1),
            torch.where((lb >= 0) & (lb < n), 1 - f, torch.zeros_like(f)),
            torch.where((lb >= -1) & (lb < n - 1), f, torch.zeros_like(f)))


def _back64(G, P, theta, out):
    """out[z][y][x] += the depth-weighted bilinear back projection of P [i][j]."""
    s = G.source(theta)
    x1 = G.x_p0 + (torch.arange(G.nx, dtype=torch.float64, device="cuda") + 0.5) * G.vx
    y1 = G.y_p0 + (torch.arange(G.ny, dtype=torch.float64, device="cuda") + 0.5) * G.vy
    s2 = s[0] ** 2 + s[1] ** 2 + s[2] ** 2
    for z in range(G.nz):
        z1 = G.z_p0 + (z + 0.5) * G.vz
        t = (-G.detectorR - s[2]) / (z1 - s[2])
        c0, c1, w0, w1 = _taps64((s[0] + (x1 - s[0]) * t - G.x_d0) / G.bx, G.nbx)
        r0, r1, v0, v1 = _taps64((s[1] + (y1 - s[1]) * t - G.y_d0) / G.by, G.nby)
        q = P[c0] * w0[:, None] + P[c1] * w1[:, None]          # [x][j]
        u = q[:, r0] * v0 + q[:, r1] * v1                      # [x][y]
        dist = ((s[0] - x1) ** 2)[:, None] + ((s[1] - y1) ** 2)[None, :] + (s[2] - z1) ** 2
        out[z] += (u * (G.vz * s2) / dist).t()


def _omega64(pot, t, delta):
    a = t.abs() / delta
    if pot == "q2":
        return torch.ones_like(t)
    if pot == "lange":
        return 1.0 / (1.0 + a)
    if pot == "hyperbola":
        return 1.0 / torch.sqrt(1.0 + a * a)
    return 1.0 / a.clamp_min(1.0)


def _prior64(x, pot, delta, zr):
    """RDD, RD of the 26 neighbours; a neighbour outside counts as a difference of 0."""
    offs = [(z, y, q) for z in (-1, 0, 1) for y in (-1, 0, 1) for q in (-1, 0, 1)
            if (z, y, q) != (0, 0, 0)]
    w = {o: 1.0 / math.sqrt(o[1] ** 2 + o[2] ** 2 + (o[0] * zr) ** 2) for o in offs}
    rdd = torch.full_like(x, sum(w.values()))
    rd = torch.zeros_like(x)
    for o in offs[13:]:  # one of each pair of opposite neighbours
        a = tuple(slice(max(0, -k), n - max(0, k)) for k, n in zip(o, x.shape))
        b = tuple(slice(max(0, k), n + min(0, k)) for k, n in zip(o, x.shape))
        t = x[a] - x[b]
        om = _omega64(pot, t, delta)
        rdd[a] += w[o] * (om - 1.0)
        rdd[b] += w[o] * (om - 1.0)
        om = om * t * w[o]
        rd[a] += om
        rd[b] -= om
    return rdd, rd


def _f32(v):
    return float(np.float32(v))


def _ostr64(c, i, x):
    """The OSTR iterations from x [z][y][x] (float64), the counts as given."""
    G = _Geo(i["g"])
    A, M = c["views"], c["subsets"]
    V = [None if t is None else t.view(A, G.nbx, G.nby) for t in (i["y"], i["b"], i["r"])]
    y, b, r = (None if t is None else (lambda a, t=t: t[a].double()) for t in V)
    d = torch.zeros_like(x)
    bx, by = G.bins()
    for a in range(A):
        s = G.source(i["angles"][a])
        hit = _hits64(G, i["angles"][a])
        L = torch.sqrt((bx - s[0])[:, None] ** 2 + (by - s[1])[None, :] ** 2
                       + (G.detectorR + s[2]) ** 2)
        ya = y(a)
        dif = ya - (r(a) if r else 0.0)
        dif = torch.where(dif <= 0, ya, dif)
        yry = torch.where(ya != 0, dif * dif / torch.where(ya != 0, ya, torch.ones_like(ya)),
                          torch.zeros_like(ya))
        _back64(G, yry * L * hit, i["angles"][a], d)
    order = _order(A, M)
    vs = A // M
    beta, delta = _f32(c["beta"]), _f32(c["delta"])
    for _ in range(c["iters"]):
        for m in range(M):
            cap = torch.zeros_like(x)
            for a in order[m * vs:(m + 1) * vs]:
                a = int(a)
                th = i["angles"][a]
                line, _ = _project64(G, x.view(-1), th)
                yb = b(a) * torch.exp(-line * math.cos(float(th)))
                h = (y(a) / (yb + (r(a) if r else 0.0)) - 1.0) * yb
                _back64(G, h, th, cap)
            rdd, rd = _prior64(x, c["potential"], delta, G.vz / G.vx)
            x = (x - (M * cap + beta * rd) / (d + 2.0 * beta * rdd)).clamp_min(0.0)
    return x


def _hits64(G, theta):
    """1 for the rays [i][j] of a view that meet the volume, else 0."""
    s = G.source(theta)
    bx, by = G.bins()
    lo = torch.full((G.nbx, G.nby), -1e300, dtype=torch.float64, device="cuda")
    hi = -lo
    dz = torch.tensor(-G.detectorR - s[2], dtype=torch.float64, device="cuda")
    for dk, p, n, v, o in (((bx - s[0])[:, None], G.x_p0, G.nx, G.vx, s[0]),
                           ((by - s[1])[None, :], G.y_p0, G.ny, G.vy, s[1]),
                           (dz, G.z_p0, G.nz, G.vz, s[2])):
        dk = torch.where(dk == 0, torch.full_like(dk, 1e-30), dk)
        a0, a1 = (p - o) / dk, (p + n * v - o) / dk
        lo = torch.maximum(lo, torch.minimum(a0, a1))
        hi = torch.minimum(hi, torch.maximum(a0, a1))
    return (lo < hi).double()


def _ossart64(c, i):
    G = _Geo(i["g"])
    A, M = c["views"], c["subsets"]
    vs, sub = A // M, 2 if c["supersample"] else 1
    p = torch.log(i["b"] / i["y"].clamp_min(1.0)).view(A, G.nbx, G.nby)
    x = i["x0"].double().view(G.nz, G.ny, G.nx)
    order = _order(A, M)
    lam, beta, delta = _f32(0.8), _f32(c["beta"]), _f32(c["delta"])

    def merge(t):
        if sub == 1:
            return t
        return (t[0::2, 0::2] + t[1::2, 0::2] + t[0::2, 1::2] + t[1::2, 1::2]) * 0.25

    for _ in range(c["iters"]):
        for m in range(M):
            u, sens = torch.zeros_like(x), torch.zeros_like(x)
            for a in order[m * vs:(m + 1) * vs]:
                th = i["angles"][int(a)]
                est, norm = (merge(t) for t in _project64(G, x.reshape(-1), th, sub))
                if c["cos"]:
                    est = est * math.cos(float(th))
                diff = torch.where(norm != 0, (p[int(a)].double() - est)
                                   / torch.where(norm != 0, norm, torch.ones_like(norm)),
                                   torch.zeros_like(norm))
                _back64(G, diff, th, u)
                _back64(G, torch.ones_like(diff), th, sens)
            if c["regularized"]:
                u = u + beta * _prior64(x, "hyperbola", delta, 1.0)[1]
            ok = sens != 0
            x = (x + lam * torch.where(ok, u / torch.where(ok, sens, torch.ones_like(sens)),
                                       torch.zeros_like(u))).clamp_min(0.0)
    return x.view(-1)


def _calls64(c, i):
    G = _Geo(i["g"])
    A, M = c["views"], c["subsets"]
    vs = A // M
    order = _order(A, M)
    x = i["x0"].double().view(G.nz, G.ny, G.nx)
    cap = torch.zeros_like(x)
    lines, hs = [], []
    for a in order[vs:2 * vs]:
        th = i["angles"][int(a)]
        line = _project64(G, x.view(-1), th)[0] * math.cos(float(th))
        yb = i["b"].view(A, G.nbx, G.nby)[int(a)].double() * torch.exp(-line)
        h = (i["y"].view(A, G.nbx, G.nby)[int(a)].double() / yb - 1.0) * yb
        _back64(G, h, th, cap)
        lines.append(line.view(-1))
        hs.append(h.view(-1))
    cap *= M
    rdd, rd = _prior64(x, c["potential"], _f32(c["delta"]), _f32(i["g"].z_xy_ratio))
    d = (float(c["I0"]) * 600.0 * 0.3 * A * (0.5 + i["x0"])).double().view(x.shape)
    beta = _f32(c["beta"])
    new = (x - (cap + beta * rd) / (d + 2.0 * beta * rdd)).clamp_min(0.0)
    return [torch.cat(lines), torch.cat(hs)] + [t.reshape(-1) for t in (cap, rdd, rd, new)]


def _psi64(pot, t, delta):
    a = t.abs() / delta
    if pot == "q2":
        return 0.5 * t * t
    if pot == "lange":
        return delta * delta * (a - torch.log1p(a))
    if pot == "hyperbola":
        return delta * delta * (a * a / (torch.sqrt(1.0 + a * a) + 1.0))
    return torch.where(a <= 1.0, 0.5 * t * t, delta * t.abs() - 0.5 * delta * delta)


def _objective64(c, i):
    G = _Geo(i["g"])
    A = c["views"]
    x = i["x0"].double().view(G.nz, G.ny, G.nx)
    data = 0.0
    for a in range(A):
        th = i["angles"][a]
        line = _project64(G, x.view(-1), th)[0] * math.cos(float(th))
        m = i["b"].view(A, G.nbx, G.nby)[a].double() * torch.exp(-line)
        y = i["y"].view(A, G.nbx, G.nby)[a].double()
        data += float((m - torch.where(y > 0, y * torch.log(m), torch.zeros_like(y))).sum())
    delta, zr = _f32(c["delta"]), G.vz / G.vx
    pen = 0.0
    for o in [(z, y, q) for z in (-1, 0, 1) for y in (-1, 0, 1) for q in (-1, 0, 1)][14:]:
        a = tuple(slice(max(0, -k), n - max(0, k)) for k, n in zip(o, x.shape))
        b = tuple(slice(max(0, k), n + min(0, k)) for k, n in zip(o, x.shape))
        w = 1.0 / math.sqrt(o[1] ** 2 + o[2] ** 2 + (o[0] * zr) ** 2)
        pen += w * float(_psi64(c["potential"], x[a] - x[b], delta).sum())
    return [data, pen]


def _net64(net):
    """The network's weights as conv3d tensors [out][in][dz][dy][dx] and biases."""
    p = net.params.double()
    o, W, B = 0, [], []
    for ni, no in ((1, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 1)):
        w = p[o:o + 27 * no * ni].view(3, 3, 3, no, ni).permute(3, 4, 0, 1, 2).contiguous()
        o += 27 * no * ni
        W.append(w)
        B.append(p[o:o + no].clone())
        o += no
    return W, B


def _conv64(a, w, b):
    """conv3d as 27 matrix products (float64 tensors [patch][channel][z][y][x])."""
    nb, ni, nz, ny, nx = a.shape
    pad = F.pad(a, (1, 1, 1, 1, 1, 1))
    out = b.view(1, -1, 1, 1, 1).expand(nb, -1, nz, ny, nx)
    for t in range(27):
        z, y, q = t // 9, (t // 3) % 3, t % 3
        out = out + torch.einsum("oi,bizyx->bozyx", w[:, :, z, y, q],
                                 pad[:, :, z:z + nz, y:y + ny, q:q + nx])
    return out


def _forward64(W, B, x, s):
    a = (s * x)[:, None]
    for k in range(5):
        a = torch.relu(_conv64(a, W[k], B[k]))
    return _conv64(a, W[5], B[5])[:, 0]


def _cnn64(c, st):
    nx, ny, nz, nb = st["dims"]
    if nx * ny * nz * nb > 1_200_000:  # the layers in 64 bits take too long beyond this
        return None
    net = st["net"]
    W, B = _net64(net)
    x = st["x"].double().view(nb, nz, ny, nx)
    if c["kind"] == "cnn_forward":
        f = _forward64(W, B, x, net.scale)
        return (x + f / net.scale).clamp_min(0.0).view(-1)
    leaves = [t.requires_grad_(True) for t in W + B]
    t = st["t"].double().view(x.shape)
    loss, n = 0.0, x.numel()
    for k in range(nb):  # one patch at a time: the saved layers of one patch fit easily
        f = _forward64(W, B, x[k:k + 1], net.scale)
        part = ((f - net.scale * (t[k:k + 1] - x[k:k + 1])) ** 2).sum() / n
        part.backward()
        loss += float(part.detach())
    out = []
    for w, b in zip(leaves[:6], leaves[6:]):
        out += [w.grad.permute(2, 3, 4, 0, 1).reshape(-1), b.grad.view(-1)]
    return [loss, torch.cat(out)]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("cnn_forward", "cnn_grad"):
        return _cnn64(c, prepare(c, seed))
    if kind == "dual":
        st = prepare(c, seed)
        he, le = st["he"].double(), st["le"].double()
        if st["level"] is not None:
            m = he > st["level"]
            he, le = he * m, le * m
        return [torch.stack([he - le * w for w in st["w"]])] + [None] * len(st["w"])
    if kind == "batch":
        out = []
        for k, s in enumerate(_batch_cases(c, seed)):
            i = _inputs(s, seed * 10 + k)
            out.append(_ostr64(s, i, i["x0"].double().view(s["nz"], s["ny"], s["nx"])).view(-1))
        return out
    i = _inputs(c, seed)
    if kind == "recon":
        x = torch.zeros(c["nz"], c["ny"], c["nx"], dtype=torch.float64, device="cuda")
        return _ostr64(c, i, x).view(-1)
    if kind == "iterate":
        return _ostr64(c, i, i["x0"].double().view(c["nz"], c["ny"], c["nx"])).view(-1)
    if kind == "ossart":
        return _ossart64(c, i)
    if kind == "calls":
        return _calls64(c, i)
    return _objective64(c, i)

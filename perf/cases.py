"""Performance cases of the step loop, through the Python binding.

A case is one run as a user's program makes it: the particles of a release or
of a saved state go in, the t = 0 pass and the steps up to an output frame
run, and the frame's particles (and, where asked for, the maxima maps) come
out. Three entry points carry the work: `Slab` (one scenario, FP32_SPLIT or
FP64_PLAIN), `Batch` (an ensemble on one terrain) and `Server` (a burst of
requests to a running server). Sizes are those of this repository's workloads
(slab-pro_b200/workloads.py): 1 600 particles on the 35-degree slope, served
requests around 20 000, ensemble members of 1.9 k to 265 k at 2 m, the 0.6 M
Voellmy case at 1 m, served requests up to 2 M and the 12 M ellipse on the
8192^2 DEM at 0.5 m; terrains are the fractal slopes of the same construction,
built on the GPU from the seed, most of them with odd sizes.

The seed sets the terrain's roughness, the release height and, for a saved
state, the particles; the release outlines belong to the case, so that every
seed has the same number of particles.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "slab-pro_b200"))

import slab  # noqa: E402

GRAVITY, CFL, DT_MAX, FLIP, FRAME_S = 9.81, 0.5, 0.01, 0.95, 1.0


# ------------------------------------------------------------------- cases


def _one(name, kind, prec, nx, ny, dx, a, b, rot, law, rho, frames, maps, per_cell=4.0):
    """One scenario. kind: "box" or "release" (a rectangle or an ellipse of
    half axes a x b cells, sampled 2 x 2 per cell) or "saved" (particles in
    motion over a tongue a cells long and at most b wide, per_cell of them for
    each cell of that frame, handed over as host arrays)."""
    return {"name": name, "kind": kind, "prec": prec, "nx": nx, "ny": ny, "dx": dx, "a": a, "b": b, "rot": rot, "law": law, "rho": rho,
            "frames": frames, "maps": maps, "per_cell": per_cell}


def listed():
    return [
        # the smallest run there is: 1 600 particles on the 35-degree slope at
        # 5 m, Coulomb; launches and latency count. In both arithmetics.
        _one("slope35 1600 fp32", "box", "fp32", 401, 101, 5.0, 10, 10, 0.0, "COULOMB", 300.0, 5, True),
        _one("slope35 1600 fp64", "box", "fp64", 401, 101, 5.0, 10, 10, 0.0, "COULOMB", 300.0, 5, True),
        # a served request of the median size (20 k particles) run alone, mu(I)
        _one("request 20k fp32", "release", "fp32", 1203, 901, 0.5, 52.3, 30.7, 33.0, "MU_I", 1500.0, 3, False),
        # a large ensemble member run alone: 2 m, Voellmy
        _one("member 180k fp32", "release", "fp32", 2047, 1801, 2.0, 141.3, 101.9, 71.0, "VOELLMY", 300.0, 3, True),
        # a developed flow: a stretched tongue with a thin tail, most tiles with
        # few particles, resumed from a saved state
        _one("thin tail 300k fp32", "saved", "fp32", 2501, 2003, 1.0, 1400.0, 520.0, 0.0, "VOELLMY", 300.0, 2, True, 0.413),
        # the 0.6 M case at 1 m, dense and irregular, resumed from a saved state; in both arithmetics
        _one("tongue 637k fp32", "saved", "fp32", 2501, 1903, 1.0, 700.0, 240.0, 0.0, "VOELLMY", 300.0, 2, True, 3.79),
        _one("tongue 637k fp64", "saved", "fp64", 2501, 1903, 1.0, 700.0, 240.0, 0.0, "VOELLMY", 300.0, 1, True, 3.79),
        # the largest served request: 2 M particles at 0.5 m, Coulomb; in both arithmetics
        _one("request 2M fp32", "release", "fp32", 4001, 3003, 0.5, 505.0, 315.0, 12.0, "COULOMB", 1500.0, 2, False),
        _one("request 2M fp64", "release", "fp64", 3001, 2003, 0.5, 505.0, 315.0, 12.0, "COULOMB", 1500.0, 1, False),
        # the headline run: 12 M particles on the 8192^2 DEM at 0.5 m, mu(I)
        _one("headline 12M fp32", "release", "fp32", 8192, 8192, 0.5, 1200.0, 800.0, 0.0, "MU_I", 1500.0, 2, False),
        # an ensemble of 16 members (1.9 k to 265 k particles) on one 2 m terrain
        {"name": "ensemble 16 fp32", "kind": "batch", "nx": 1201, "ny": 1103, "dx": 2.0, "members": 16, "shape_seed": 2028, "lo": 10.0,
         "hi": 150.0},
        # a burst of 12 requests to a running server on one 0.5 m terrain
        {"name": "served burst 12 fp32", "kind": "server", "nx": 1801, "ny": 1507, "dx": 0.5, "members": 12, "shape_seed": 2029, "lo": 20.0,
         "hi": 130.0},
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["release", "release", "release", "saved", "saved", "batch", "server"])
    if kind in ("batch", "server"):
        return {"kind": kind, "nx": rng.randint(1000, 1800), "ny": rng.randint(1000, 1600), "dx": rng.choice([0.5, 1.0, 2.0]),
                "members": rng.randint(4, 16), "shape_seed": rng.randint(0, 10**6), "lo": rng.uniform(8.0, 30.0),
                "hi": rng.uniform(60.0, 150.0)}
    prec = rng.choice(["fp32", "fp32", "fp32", "fp64"])
    if kind == "saved":
        n = math.exp(rng.uniform(math.log(5000.0), math.log(1.5e6)))
        per_cell = math.exp(rng.uniform(math.log(0.4), math.log(4.5)))
        area, aspect = n / per_cell, rng.uniform(2.0, 4.0)
        a, b = math.sqrt(area * aspect), math.sqrt(area / aspect)
        nx, ny = int(1.3 * a), int(1.6 * b)
    else:
        n = math.exp(rng.uniform(math.log(1600.0), math.log(2.2e6 if prec == "fp64" else 6e6)))
        per_cell, aspect = 4.0, rng.uniform(1.0, 2.5)
        a, b = math.sqrt(n / 4.0 * aspect / math.pi), math.sqrt(n / 4.0 / aspect / math.pi)
        nx, ny = int(2.6 * a), int(2.4 * max(a, b))
    return {"kind": kind, "prec": prec, "nx": nx + rng.randint(160, 560), "ny": ny + rng.randint(160, 460),
            "dx": rng.choice([0.5, 1.0, 2.0, 5.0]), "a": a, "b": b, "rot": rng.uniform(0.0, 180.0) if kind == "release" else 0.0,
            "law": rng.choice(["COULOMB", "VOELLMY", "MU_I"]), "rho": rng.choice([300.0, 1500.0]), "frames": 1, "maps": rng.random() < 0.5,
            "per_cell": per_cell}


# ------------------------------------------------------------------ inputs


def _terrain(c, seed):
    """A fractal slope (30 degrees easing to 5, fBm roughness, Hurst 0.8, no
    wavelength under 20 m or 10 nodes), or the 35-degree slope with its arc."""
    nx, ny, dx = c["nx"], c["ny"], c["dx"]
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 13)
    L = nx * dx
    x = torch.arange(nx, dtype=torch.float64, device="cuda") * dx
    if c["kind"] == "box":
        a, brk, R = math.radians(35.0), 1200.0, 100.0
        t = R * math.tan(a / 2.0)
        x1, x2 = brk - t * math.cos(a), brk + t
        zx = torch.where(x <= x1, math.tan(a) * (brk - x),
                         torch.where(x < x2, R - torch.sqrt(torch.clamp(R * R - (x - x2) ** 2, min=0.0)), torch.zeros_like(x)))
        rms = 0.05
    else:
        s0, s1 = math.tan(math.radians(30.0)), math.tan(math.radians(5.0))
        u = torch.clamp((x - 0.6 * L) / (0.12 * L), 0.0, 1.0)
        slope = s0 + (s1 - s0) * (u * u * (3 - 2 * u))
        zx = torch.zeros_like(x)
        zx[1:] = -torch.cumsum(0.5 * (slope[1:] + slope[:-1]) * dx, 0)
        zx = zx - zx.min()
        rms = min(7.5, L / 500.0)
    kx = torch.fft.fftfreq(nx, d=dx, dtype=torch.float64, device="cuda")
    ky = torch.fft.rfftfreq(ny, d=dx, dtype=torch.float64, device="cuda")
    K = torch.sqrt(kx[:, None] ** 2 + ky[None, :] ** 2)
    amp = torch.where(K > 0, K, torch.ones_like(K)) ** -1.8
    amp[(K > 1.0 / max(20.0, 10.0 * dx)) | (K < 1.0 / max(nx * dx, ny * dx))] = 0.0
    del kx, ky, K
    ph = torch.complex(torch.randn(amp.shape, dtype=torch.float64, device="cuda", generator=g),
                       torch.randn(amp.shape, dtype=torch.float64, device="cuda", generator=g))
    rough = torch.fft.irfft2(amp * ph, s=(nx, ny))
    del amp, ph
    rough *= rms / rough.std()
    return zx[:, None] + rough


def _cfg(law, rho, total_time, u=0.5):
    cfg = dict(gravity=GRAVITY, rho=rho, C_cfl=CFL, dt_max=DT_MAX, flip_ratio=FLIP, output_dt=FRAME_S, total_time=total_time, friction=law)
    if law == "COULOMB":
        cfg["coulomb_mu"] = 0.3 + 0.2 * u
    elif law == "VOELLMY":
        cfg.update(voellmy_mu=0.1 + 0.3 * u, voellmy_xi=500.0 + 2000.0 * u)
    else:
        cfg.update(mui_mu1=0.38, mui_mu2=0.64, mui_I0=0.279, mui_d=5e-4, mui_phi=0.6)
    return cfg


def _release(c, h0):
    dx = c["dx"]
    if c["kind"] == "box":
        return {"type": "RECTANGLE", "center": (150.0, 250.0), "Lx": 2 * c["a"] * dx, "Ly": 2 * c["b"] * dx, "rotation_deg": 0.0, "h0": h0}
    big = max(c["a"], c["b"]) + 8
    return {"type": "ELLIPSE", "center": ((big + 0.05 * c["nx"]) * dx, 0.5 * c["ny"] * dx), "rx": c["a"] * dx, "ry": c["b"] * dx,
            "rotation_deg": c["rot"], "h0": h0}


def _members(c, seed):
    """The scenarios of an ensemble or a burst: outlines from the case, heights and friction from the seed."""
    shape, u = np.random.default_rng(c["shape_seed"]), np.random.default_rng(seed + 77)
    dx, out = c["dx"], []
    for k in range(c["members"]):
        ra, rb = np.exp(shape.uniform(math.log(c["lo"]), math.log(c["hi"]), 2))
        rot, big = shape.uniform(0.0, 180.0), max(ra, rb) + 12.0
        cx, cy = shape.uniform(big, max(big + 1.0, c["nx"] / 3.0)), shape.uniform(big, c["ny"] - big)
        law = "VOELLMY" if c["kind"] == "batch" else ["COULOMB", "VOELLMY", "MU_I"][k % 3]
        rel = {"type": "ELLIPSE", "center": (float(cx * dx), float(cy * dx)), "rx": float(ra * dx), "ry": float(rb * dx),
               "rotation_deg": float(rot), "h0": float(u.uniform(0.5, 3.0))}
        out.append((_cfg(law, 300.0 if c["kind"] == "batch" else 1500.0, FRAME_S, float(u.uniform(0.0, 1.0))), rel))
    return out


def _saved(c, seed):
    """A tongue in motion, dense at the front and thinning out to its tail and
    sides, heights and velocities varying along it; in the order of its cells."""
    g = torch.Generator(device="cuda").manual_seed(seed * 104729 + 5)
    dx, a, b = c["dx"], c["a"], c["b"]
    n = int(c["per_cell"] * a * b)
    r = torch.rand((3, n), dtype=torch.float64, device="cuda", generator=g)
    gn = torch.randn((3, n), dtype=torch.float64, device="cuda", generator=g)
    u = torch.sqrt(r[0])  # denser towards the front
    y = torch.clamp(gn[0] * 0.4, -1.0, 1.0) * (0.35 + 0.65 * u)
    X, Y = (0.06 * c["nx"] + 10.3 + a * u) * dx, (0.5 * c["ny"] + 0.5 * b * y) * dx
    order = torch.argsort(torch.floor(X / dx) * c["ny"] + torch.floor(Y / dx), stable=True)
    h = (0.4 + 2.2 * u * (1.0 - y * y)) * (0.9 + 0.2 * r[1])
    A = torch.full_like(h, dx * dx / 4.0) * (0.8 + 0.4 * r[2])
    P = {"x": torch.stack([X, Y], 1)[order], "v": torch.stack([6.0 + 9.0 * u + 0.2 * gn[1], 0.6 * y + 0.2 * gn[2]], 1)[order],
         "h": h[order], "A": A[order], "mass": (c["rho"] * h * A)[order]}
    P["vz"] = torch.zeros_like(P["h"])
    P["z"] = torch.zeros_like(P["h"])
    return P


def _h0(seed):
    return 1.5 + 1.5 * float(np.random.default_rng(seed + 31).random())


def prepare(case, seed):
    z = _terrain(case, seed).cpu().numpy()
    dx = case["dx"]
    if case["kind"] == "batch":
        return {"case": case, "z": z, "members": _members(case, seed)}
    if case["kind"] == "server":
        return {"case": case, "server": slab.Server(z, dx, max_scenarios=16), "members": _members(case, seed)}
    s = slab.Slab(z, dx)
    s.set_params(_cfg(case["law"], case["rho"], case["frames"] * FRAME_S), slab.FP64_PLAIN if case["prec"] == "fp64" else slab.FP32_SPLIT)
    st = {"case": case, "slab": s}
    if case["kind"] == "saved":
        st["particles"] = {k: v.cpu().numpy() for k, v in _saved(case, seed).items()}
    else:
        st["release"] = _release(case, _h0(seed))
    return st


# --------------------------------------------------------------------- run


def _hazard(shape, boxes):
    """The ensemble's hazard maps as float32 rasters: the largest flow height and speed squared over all members."""
    H, V = np.zeros(shape, np.float32), np.zeros(shape, np.float32)
    for (i0, i1, j0, j1), hm, vm in boxes:
        if i1 >= i0 and j1 >= j0:
            w = (slice(i0, i1 + 1), slice(j0, j1 + 1))
            H[w] = np.maximum(H[w], hm)
            V[w] = np.maximum(V[w], vm)
    return {"h_max": H, "v_max2": V}


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        b = slab.Batch(state["z"], c["dx"], c["members"])
        ids = [b.add_release(cfg, rel) for cfg, rel in state["members"]]
        b.run()
        out = _hazard(state["z"].shape, [b.max_box(k) for k in ids])
        parts = [b.particles(k) for k in ids]
        b.close()
        out["particles"] = _flat(parts)
        return out
    if c["kind"] == "server":
        s = state["server"]
        ids = [s.submit_release(cfg, rel) for cfg, rel in state["members"]]
        s.drain()
        res = [s.result(k) for k in ids]
        out = _hazard((c["nx"], c["ny"]), [(r["box"], r["h_max"], r["v_max2"]) for r in res])
        out["particles"] = _flat(res)
        return out
    s = state["slab"]
    if c["kind"] == "saved":
        s.upload(state["particles"])
    else:
        s.upload_release(state["release"])
    s.initial_pass()
    for _ in range(c["frames"]):
        s.advance_to_frame()
    if c["prec"] == "fp64":
        out = {"particles": s.particles()}  # all the digits that the arithmetic has
        if c["maps"]:
            out["h_max"], out["v_max2"] = s.max_maps()
        return out
    s.frame_capture(0)
    out = {"particles": s.frame_wait(0)["particles"]}  # float32, as in the frame's PLY file
    if c["maps"]:
        hm, vm = s.max_maps()
        out["h_max"], out["v_max2"] = hm.astype(np.float32), vm.astype(np.float32)  # as in the GeoTIFF of the maxima
    return out


def _flat(parts):
    """The members' particles one after the other, float32 as in a PLY file."""
    return np.concatenate([np.concatenate([p["x"], p["v"], p["h"][:, None], p["mass"][:, None]], 1).astype(np.float32) for p in parts])


# -------------------------------------------------------------------- work


def _np_of(c):
    if c["kind"] == "box":
        return 16.0 * c["a"] * c["b"]
    if c["kind"] == "release":
        return 4.0 * math.pi * c["a"] * c["b"]
    return c["per_cell"] * c["a"] * c["b"]


def work(case):
    """Per particle and step, FP32: P2G reads the state (28 bytes: cell,
    offset, velocity, height, mass), G2P reads and writes what moves (24 each
    way); per active node 124 bytes (sums written and read, terrain, velocity
    written and read, maxima). FP64: 128 and 248. About 420 operations per
    particle-step (two 9-node stencils) and 60 per node. Once per run: the
    particles in (32 bytes each, 80 as FP64 host arrays) and out."""
    c = case
    if c["kind"] in ("batch", "server"):
        n = sum(4.0 * math.pi * rel["rx"] * rel["ry"] / c["dx"] ** 2 for _, rel in _members(c, 0))
        steps, fp64, once = 100, False, 32 + 48
    else:
        n, steps, fp64 = _np_of(c), 100 * c["frames"], c["prec"] == "fp64"
        once = (80 if c["kind"] == "saved" else 32) + (80 if fp64 else 32)
    nodes = 0.6 * c["a"] * c["b"] if c["kind"] == "saved" else 0.26 * n
    per = (128, 248) if fp64 else (76, 124)
    return {"bytes": steps * (per[0] * n + per[1] * nodes) + once * n, "flops": steps * (420 * n + 60 * nodes)}


# ------------------------------------------------------------------- exact


def _samples(rel, dx):
    """The 2 x 2 samples per cell inside the outline, in the order of the cells (j fastest), then of the four displacements."""
    ood = 1.0 / dx
    cx, cy = rel["center"]
    if rel["type"] == "RECTANGLE":
        half, area = math.sqrt(rel["Lx"] ** 2 + rel["Ly"] ** 2) / 2.0, rel["Lx"] * rel["Ly"]
    else:
        half, area = max(rel["rx"], rel["ry"]), math.pi * rel["rx"] * rel["ry"]
    x0, x1 = math.floor((cx - half) * ood) * dx, math.ceil((cx + half) * ood) * dx
    y0, y1 = math.floor((cy - half) * ood) * dx, math.ceil((cy + half) * ood) * dx
    nx, ny = int(round((x1 - x0) * ood)), int(round((y1 - y0) * ood))
    i = torch.arange(nx, dtype=torch.float64, device="cuda")
    j = torch.arange(ny, dtype=torch.float64, device="cuda")
    ox = torch.tensor([0.25, 0.75, 0.25, 0.75], dtype=torch.float64, device="cuda")
    oy = torch.tensor([0.25, 0.25, 0.75, 0.75], dtype=torch.float64, device="cuda")
    X = (((i[:, None] + ox) * dx + x0)[:, None, :]).expand(nx, ny, 4).reshape(-1)
    Y = (((j[:, None] + oy) * dx + y0)[None, :, :]).expand(nx, ny, 4).reshape(-1)
    rot = rel["rotation_deg"] * math.pi / 180.0
    c, s = math.cos(-rot), math.sin(-rot)
    px, py = X - cx, Y - cy
    lx, ly = c * px - s * py, s * px + c * py
    if rel["type"] == "RECTANGLE":
        keep = (lx.abs() <= rel["Lx"] / 2.0) & (ly.abs() <= rel["Ly"] / 2.0)
    else:
        keep = (lx / rel["rx"]) ** 2 + (ly / rel["ry"]) ** 2 <= 1.0
    return torch.stack([X[keep], Y[keep]], 1), area


def _released(rel, dx, rho):
    x, area = _samples(rel, dx)
    n, h0 = len(x), rel["h0"]
    A = torch.full((n,), area * h0 / (n * h0), dtype=torch.float64, device="cuda")
    h = torch.full_like(A, h0)
    return {"x": x, "v": torch.zeros_like(x), "vz": torch.zeros_like(h), "h": h, "A": A, "mass": rho * h * A, "z": torch.zeros_like(h)}


def _weights(f):
    """Quadratic B-spline weights and derivatives of the nodes at distances f, f - 1, f - 2 (f in [0.5, 1.5))."""
    w = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1.0) ** 2, 0.5 * (f - 0.5) ** 2]
    return w, [f - 1.5, -2.0 * (f - 1.0), f - 0.5]


def _simulate(z, dx, cfg, P, frames):
    """The depth-averaged MPM step loop in FP64: P2G, grid update with friction, G2P; until `frames` output frames are done."""
    nx, ny = z.shape
    gx, gy = torch.zeros_like(z), torch.zeros_like(z)
    gx[:-1, :-1] = (z[1:, :-1] + z[1:, 1:] - z[:-1, :-1] - z[:-1, 1:]) / 2.0 / dx
    gy[:-1, :-1] = (z[:-1, 1:] + z[1:, 1:] - z[:-1, :-1] - z[1:, :-1]) / 2.0 / dx
    ct = 1.0 / torch.sqrt(1.0 + gx * gx + gy * gy)
    x, v, vz, h, A, m, zp = (P[k].clone() for k in ("x", "v", "vz", "h", "A", "mass", "z"))
    hmax, vmax2 = torch.zeros_like(z), torch.zeros_like(z)
    g, rho, law, fr = cfg["gravity"], cfg["rho"], cfg["friction"], cfg["flip_ratio"]
    t, frame, first = 0.0, 0, True
    while first or frame < frames:
        # dt from the fastest particle, cut at the next frame; the t = 0 pass has none
        frame_end = False
        if first:
            dt = 0.0
        else:
            speed = float((v * v).sum(1).max().sqrt())
            dt = min(cfg["C_cfl"] * dx / speed, cfg["dt_max"]) if speed > 0 else cfg["dt_max"]
            nxt = cfg["output_dt"] * (frame + 1)
            if t + dt > nxt - 1e-12:
                dt = nxt - t
            frame_end = nxt - (t + dt) < 1e-13
        # the nodes that the particles reach
        lo, hi = (x.min(0).values / dx).floor().long() - 2, (x.max(0).values / dx).floor().long() + 4
        i0, j0, i1, j1 = (int(k) for k in (lo[0], lo[1], hi[0], hi[1]))
        i0, j0, i1, j1 = max(i0, 0), max(j0, 0), min(i1, nx), min(j1, ny)
        W, box = j1 - j0, (slice(i0, i1), slice(j0, j1))
        u = x / dx
        base = torch.floor(u - 0.5)
        wx, dwx = _weights(u[:, 0] - base[:, 0])
        wy, dwy = _weights(u[:, 1] - base[:, 1])
        node0 = (base[:, 0].long() - i0) * W + (base[:, 1].long() - j0)
        cell = u.floor().long()
        cx, cy, cc = gx[cell[:, 0], cell[:, 1]], gy[cell[:, 0], cell[:, 1]], ct[cell[:, 0], cell[:, 1]]
        pull = m * g * cc * cc
        press = 0.5 * rho * g * cc * cc * h * h * A / dx
        q = torch.stack([m, m * v[:, 0], m * v[:, 1], m * h], 1)
        acc = torch.zeros(((i1 - i0) * W, 6), dtype=torch.float64, device=z.device)
        for a in range(3):
            for b in range(3):
                w = wx[a] * wy[b]
                on = (w > 3e-3).double()
                w = w * on
                c = torch.empty((len(w), 6), dtype=torch.float64, device=z.device)
                c[:, :4] = q * w[:, None]
                c[:, 4] = press * dwx[a] * wy[b] * on - pull * cx * w
                c[:, 5] = press * dwy[b] * wx[a] * on - pull * cy * w
                acc.index_add_(0, node0 + a * W + b, c)
        mi, px, py, hm, fx, fy = (acc[:, k].reshape(i1 - i0, W) for k in range(6))
        act = mi > 1e-6
        ms = torch.where(act, mi, torch.ones_like(mi))
        hn = torch.where(act, hm / ms, torch.zeros_like(mi))
        vox, voy = px / ms, py / ms
        vtx, vty = vox + dt * fx / ms, voy + dt * fy / ms
        vsq = vtx * vtx + vty * vty
        nc = ct[box]
        v3sq = vsq + (vtx * gx[box] + vty * gy[box]) ** 2
        v3 = torch.sqrt(v3sq)
        hs = torch.where(act, hn, torch.ones_like(hn))
        if law == "COULOMB":
            fric = cfg["coulomb_mu"] * g * nc
        elif law == "VOELLMY":
            fric = cfg["voellmy_mu"] * g * nc + g * v3sq / (cfg["voellmy_xi"] * hs * nc)
        else:
            In = 5.0 * cfg["mui_d"] * v3 / (2.0 * hs * nc * nc * torch.sqrt(g * hs * cfg["mui_phi"]))
            fric = (cfg["mui_mu1"] + (cfg["mui_mu2"] - cfg["mui_mu1"]) / (1.0 + cfg["mui_I0"] / In)) * g * nc
        moves = act & (vsq > 1e-16) & (dt * fric < v3)
        f = torch.where(moves, 1.0 - dt * fric / torch.where(moves, v3, torch.ones_like(v3)), torch.zeros_like(v3))
        nvx, nvy = vtx * f, vty * f
        flx, fly = torch.where(act, nvx - vox, 0.0 * vox), torch.where(act, nvy - voy, 0.0 * voy)
        hmax[box] = torch.maximum(hmax[box], hn)
        vmax2[box] = torch.maximum(vmax2[box], torch.where(act, nvx * nvx + nvy * nvy, torch.zeros_like(nvx)))
        if first:
            first = False
            continue
        n4 = torch.stack([nvx.reshape(-1), nvy.reshape(-1), flx.reshape(-1), fly.reshape(-1), z[box].reshape(-1)], 1)
        got = torch.zeros((len(h), 5), dtype=torch.float64, device=z.device)
        div = torch.zeros_like(h)
        for a in range(3):
            for b in range(3):
                k = n4[node0 + a * W + b]
                got += k * (wx[a] * wy[b])[:, None]
                div += (dwx[a] * wy[b] * k[:, 0] + dwy[b] * wx[a] * k[:, 1]) / dx
        v = fr * (v + got[:, 2:4]) + (1.0 - fr) * got[:, :2]
        zp = got[:, 4]
        vz = v[:, 0] * cx + v[:, 1] * cy
        x = x + dt * got[:, :2]
        h = h / (1.0 + dt * div)
        A = m / (h * rho)
        t += dt
        frame += int(frame_end)
    return {"x": x, "v": v, "vz": vz, "h": h, "A": A, "mass": m, "z": zp}, hmax, vmax2


def exact(case, seed):
    c, dx = case, case["dx"]
    z = _terrain(c, seed)
    if c["kind"] in ("batch", "server"):
        H, V, parts = torch.zeros_like(z), torch.zeros_like(z), []
        for cfg, rel in _members(c, seed):
            p, hm, vm = _simulate(z, dx, cfg, _released(rel, dx, cfg["rho"]), 1)
            H, V = torch.maximum(H, hm), torch.maximum(V, vm)
            parts.append(torch.cat([p["x"], p["v"], p["h"][:, None], p["mass"][:, None]], 1))
        return {"h_max": H, "v_max2": V, "particles": torch.cat(parts)}
    cfg = _cfg(c["law"], c["rho"], c["frames"] * FRAME_S)
    P = _saved(c, seed) if c["kind"] == "saved" else _released(_release(c, _h0(seed)), dx, cfg["rho"])
    p, hm, vm = _simulate(z, dx, cfg, P, c["frames"])
    if c["prec"] == "fp64":
        out = {"particles": p}
    else:
        out = {"particles": torch.cat([p["x"], p["v"], p["vz"][:, None], p["z"][:, None], p["h"][:, None], p["A"][:, None]], 1)}
    if c["maps"]:
        out["h_max"], out["v_max2"] = hm, vm
    return out

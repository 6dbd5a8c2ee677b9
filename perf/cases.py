"""Timed workloads of the framework, each through the entry points a mapping program calls.

The samples are the two of the benchmark: BCC iron (86 reflections) and FCC aluminium (64), 10-70
keV, source and detector 11 mm from the sample, detectors of 68.8 mm.  Grains are balls in a cylinder,
their spots are marked by landing points of every grain, and the distance map is the exact
Euclidean one.  Inputs are made with torch and numpy from the seed alone; ``exact`` restates each result
in 64 bits from the same inputs (the fits' derivatives by complex steps).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

SIDE_MM = 68.8128          # detector side: 1024 pixels of 0.0672 mm, 2048 of 0.0336 mm
HIT = 0.5                  # a landing within this distance of a spot counts [pixel]
DEV = "cuda"


def listed():
    fe = {"lattice": "fe", "ny": 1024, "nz": 1024, "nrot": 181}
    al = {"lattice": "al", "ny": 2048, "nz": 2048, "nrot": 361}
    return [
        # the drop-in call at its smallest: a handful of orientations at one voxel, where latency counts
        {"name": "scan-few", "kind": "scan", **fe, "n_q": 8, "median": True},
        # one seed against the 2-degree cubic grid, host arrays in and out, as the MATLAB wrapper calls it
        {"name": "scan-seed", "kind": "scan", **al, "n_q": 32768, "median": True},
        # the headline: a batch of seeds, completeness and each seed's first maximum, all on the device
        {"name": "batch-al", "kind": "batch", **al, "seeds": 64, "n_q": 32768, "median": False},
        # the same entry with the reference's four columns on the smaller sample and the 3-degree grid
        {"name": "batch-fe", "kind": "batch", **fe, "seeds": 16, "n_q": 9218, "median": True},
        # growing an indexed region: one orientation over a ball of voxels, an odd detector
        {"name": "grow", "kind": "grow", "lattice": "al", "ny": 1537, "nz": 1001, "nrot": 121, "voxels": 9171},
        # candidates competing for waiting voxels, the reference's 30,000-voxel chunk
        {"name": "compete", "kind": "compete", **al, "voxels": 30000},
        # whole indexing of some seeds: scan, top rows, local refine, Nelder-Mead fit, final scoring
        {"name": "index", "kind": "index", **fe, "seeds": 4, "n_q": 9218, "top": 400},
        # pairing of simulated and measured spots for the centre fits
        {"name": "pair", "kind": "pair", **fe, "trials": 1536},
        # orientation and centre of many grains from their matched spots, two steps
        {"name": "grains", "kind": "grains", **fe, "grains": 5000, "iters": 2},
        # the ten geometry parameters from many starts, one step
        {"name": "geometry", "kind": "geometry", **al, "grains": 500, "starts": 64},
        # residuals and their derivatives alone, for a caller's own solver
        {"name": "jacobian", "kind": "jacobian", **fe, "spots": 1000003, "mode": 1},
        # a new data set: spot images to distance map to resident map, and the first few scores on it
        {"name": "masks", "kind": "masks", **fe, "n_q": 64},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["scan", "scan", "batch", "batch", "grow", "compete", "index", "pair", "grains", "geometry",
                       "jacobian", "masks"])
    c = {"kind": kind, "lattice": rng.choice(["fe", "al"]), "ny": log(256, 2048), "nz": log(256, 2048),
         "nrot": log(37, 361)}
    if kind == "scan":
        c.update(n_q=log(1, 32768), median=rng.random() < 0.7)
    elif kind == "batch":
        c.update(seeds=log(2, 32), n_q=log(512, 32768), median=rng.random() < 0.4)
    elif kind in ("grow", "compete"):
        c.update(voxels=log(200, 30000))
    elif kind == "index":
        c.update(seeds=log(1, 4), n_q=log(1024, 9218), top=log(10, 200))
    elif kind == "pair":
        c.update(trials=log(4, 1536))
    elif kind == "grains":
        c.update(grains=log(30, 3000), iters=rng.choice([1, 2]))
    elif kind == "geometry":
        c.update(grains=log(20, 400), starts=log(1, 64))
    elif kind == "jacobian":
        c.update(spots=log(3000, 1000000), mode=rng.choice([0, 1]))
    else:
        c.update(n_q=log(1, 126))
    return c


# ---- the sample ------------------------------------------------------------------------------------

def f32(a):
    return np.ascontiguousarray(a, dtype=np.float32)


def setup(case, rng):
    """Geometry as the wrappers pass it (float32 arrays) and as 64-bit numbers rounded to float32."""
    fe = case["lattice"] == "fe"
    r = range(-4, 5)
    cand = [(h * h + k * k + l * l, h, k, l) for h in r for k in r for l in r if (h or k or l) and
            ((h + k + l) % 2 == 0 if fe else h % 2 == k % 2 == l % 2)]
    top = sorted({c[0] for c in cand})[5]
    hkl = np.array([c[1:] for c in sorted(cand) if c[0] <= top], np.float64)
    a0 = 2.8665 if fe else 4.0495
    tilt = rng.uniform(-0.5, 0.5, 3)
    ny, nz, nrot = case["ny"], case["nz"], case["nrot"]
    px = SIDE_MM / max(ny, nz)
    lss = lsd = 11.0
    tmax = math.degrees(math.acos(lsd / math.sqrt(lsd ** 2 + (0.5 * ny * px) ** 2 + (0.5 * nz * px) ** 2))) / 2
    R = rot_det(*(torch.tensor(float(t), dtype=torch.float64) for t in tilt))
    S9 = f32(np.eye(3).reshape(9))
    B9 = f32((np.eye(3) * (2 * math.pi / a0)).reshape(9))
    R9 = f32([[float(x) for x in row] for row in R]).reshape(9)
    rot = f32(np.linspace(0.0, 360.0, nrot))
    par = f32([len(hkl), nrot, lss, lsd, 0, 0, 0, 0, px, px, ny, nz, 0, 0, 0, 0, tmax, 12.39818746 / 70,
               12.39818746 / 10, 0])
    w = np.radians(rot.astype(np.float64))
    p = par.astype(np.float64)
    return {"args": (S9, B9, f32(hkl).reshape(-1), rot, R9, par), "tilt": tilt, "hkl": hkl, "b0": float(B9[0]),
            "P": {"lss": p[2], "lsd": p[3], "p0y": 0.0, "p0z": 0.0, "y00": 0.0, "z00": 0.0, "rao": 0.0,
                  "R": R9.astype(np.float64).reshape(3, 3).tolist()},
            "px": p[8], "ny": ny, "nz": nz, "tmax": p[16], "lmin": p[17], "lmax": p[18],
            "c": torch.tensor(np.cos(w), device=DEV), "s": torch.tensor(np.sin(w), device=DEV),
            "h": torch.tensor(hkl * float(B9[0]), device=DEV)}


def rot_det(tx, ty, tz):
    d = math.pi / 180
    cx, sx, cy, sy, cz, sz = (f(t * d) for t in (tx, ty, tz) for f in (torch.cos, torch.sin))
    return [[cz * cy, cz * sy * sx - sz * cx, cz * sy * cx + sz * sx],
            [sz * cy, sz * sy * sx + cz * cx, sz * sy * cx - cz * sx], [-sy, cy * sx, cy * cx]]


def quats(n, rng):
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    q[q[:, 0] < 0] *= -1
    return q


def matrices(q):
    """Rotation matrices of quaternions used as given (n x 4 tensor -> n x 3 x 3)."""
    a, b, c, d = q.unbind(-1)
    return torch.stack([2 * (a * a + b * b) - 1, 2 * (b * c - a * d), 2 * (b * d + a * c), 2 * (b * c + a * d),
                        2 * (a * a + c * c) - 1, 2 * (c * d - a * b), 2 * (b * d - a * c), 2 * (c * d + a * b),
                        2 * (a * a + d * d) - 1], -1).reshape(*q.shape[:-1], 3, 3)


def land(P, pos, g, c, s, geo):
    """Landing (u, v) and wavelength of reflections g (3 tensors, sample frame) from points pos (3 tensors) at
    rotations (c, s); everything broadcasts, real or complex."""
    R = P["R"]
    px, py, pz = pos[0], pos[1] - P["rao"], pos[2]
    swx, swy, swz = c * px - s * py, s * px + c * py, pz
    gx, gy, gz = P["lss"] + swx, swy - P["p0y"] + P["rao"], swz - P["p0z"]
    ng = torch.sqrt(gx * gx + gy * gy + gz * gz)
    kx, ky, kz = gx / ng, gy / ng, gz / ng
    L = P["lss"] + P["lsd"]
    ax = P["lsd"] - swx
    ay, az = gy * L / gx - swy, gz * L / gx - swz
    tx, ty, tz = c * g[0] - s * g[1], s * g[0] + c * g[1], g[2]
    G = torch.sqrt(tx * tx + ty * ty + tz * tz)
    x = (kx * tx + ky * ty + kz * tz) / G
    lam = -(4 * math.pi) * x / G
    s2, c2 = -2 * x * torch.sqrt(1 - x * x), 1 - 2 * x * x
    n = torch.sqrt(ty * ty + tz * tz)
    ny, nz = ty / n, tz / n
    cp = ny * ky + nz * kz
    diff = ax * ng / gx * s2 / (torch.sqrt(1 - cp * cp) * c2 - cp * s2)
    Ky, Kz = ay + diff * ny, az + diff * nz
    dx, dy, dz = swx - P["lsd"], swy - P["y00"] + P["rao"], swz - P["z00"]
    f = -(R[0][0] * dx + R[1][0] * dy + R[2][0] * dz) / (R[0][0] * ax + R[1][0] * Ky + R[2][0] * Kz)
    y2 = f * (R[0][1] * ax + R[1][1] * Ky + R[2][1] * Kz) + (R[0][1] * dx + R[1][1] * dy + R[2][1] * dz)
    z2 = f * (R[0][2] * ax + R[1][2] * Ky + R[2][2] * Kz) + (R[0][2] * dx + R[1][2] * dy + R[2][2] * dz)
    u = geo["ny"] / 2 + 0.5 - y2 / geo["px"]
    v = geo["nz"] / 2 + 0.5 - z2 / geo["px"]
    return u, v, lam, x


def landings(geo, pos, U):
    """Of trials (pos n x 3, U n x 3 x 3): selected (n, nrot, nhkl), u, v, wavelength."""
    g = torch.einsum("nij,hj->inh", U, geo["h"])[:, :, None, :]
    P3 = pos.t()[:, :, None, None]
    u, v, lam, x = land(geo["P"], P3, g, geo["c"][None, :, None], geo["s"][None, :, None], geo)
    cb = math.cos(math.radians(90 + 4 * geo["tmax"])) if 90 + 4 * geo["tmax"] <= 180 else -2.0
    ok = (x < 0) & (x > cb) & (lam > geo["lmin"]) & (lam < geo["lmax"])
    ok &= (u >= 0.5) & (u < geo["ny"] + 0.5) & (v >= 0.5) & (v < geo["nz"] + 0.5)
    return ok, u, v, lam


def per_chunk(geo):
    return max(1, int(4e7 // (geo["c"].numel() * geo["h"].shape[0])))


def sample(case, seed, spots=True):
    """Geometry, grains (quaternion, centre, radius) and the spot mask (nrot, ny, nz) of a case."""
    rng = np.random.default_rng(seed)
    geo = setup(case, rng)
    fe = case["lattice"] == "fe"
    n, rad, pts = (6, 0.05, 60) if fe else (400, 0.2, 16)
    q = quats(n, rng)
    phi, rr = rng.uniform(0, 2 * np.pi, n), rad * np.sqrt(rng.random(n))
    cen = np.stack([rr * np.cos(phi), rr * np.sin(phi), rng.uniform(-rad, rad, n)], 1)
    size = 0.55 * rad * 2 / n ** (1 / 3) * rng.lognormal(0.0, 0.0 if fe else 0.3, n)
    out = {"geo": geo, "rng": rng, "q": q, "cen": cen, "size": size, "rad": rad}
    if not spots:
        return out
    ball = rng.normal(size=(n, pts, 3))
    ball *= (rng.random((n, pts, 1)) ** (1 / 3)) / np.linalg.norm(ball, axis=2, keepdims=True)
    pos = torch.tensor((cen[:, None] + ball * size[:, None, None]).reshape(-1, 3), device=DEV)
    U = matrices(torch.tensor(q, device=DEV)).repeat_interleave(pts, 0)
    mask = torch.zeros(case["nrot"] * case["ny"] * case["nz"], dtype=torch.uint8, device=DEV)
    step = per_chunk(geo)
    for i in range(0, len(pos), step):
        ok, u, v, _ = landings(geo, pos[i:i + step], U[i:i + step])
        mask[pixel(geo, ok, u, v)] = 1
    planes = mask.view(-1, case["ny"], case["nz"])   # spots are blobs: every landing with its neighbours
    wide = planes.clone()
    wide[:, 1:] |= planes[:, :-1]
    wide[:, :-1] |= planes[:, 1:]
    planes = wide.clone()
    planes[:, :, 1:] |= wide[:, :, :-1]
    planes[:, :, :-1] |= wide[:, :, 1:]
    out["mask"] = planes.view(-1)
    return out


def pixel(geo, ok, u, v):
    """Map index of every selected landing."""
    iw = torch.arange(ok.shape[1], device=DEV)[None, :, None].expand_as(ok)[ok]
    iu, iv = torch.floor(u[ok] + 0.5).long() - 1, torch.floor(v[ok] + 0.5).long() - 1
    return (iw * geo["ny"] + iu) * geo["nz"] + iv


def distance(mask, case, most=96):
    """Squared distance of every pixel to its projection's nearest spot pixel (float32 whole numbers), exact up to
    ``most`` pixels across lines and an upper bound beyond."""
    ny, nz = case["ny"], case["nz"]
    out = torch.empty(mask.numel(), dtype=torch.float32, device=DEV)
    at = torch.arange(nz, device=DEV, dtype=torch.float32)
    far = float(4 * (ny + nz))
    planes = mask.view(-1, ny, nz)
    step = max(1, int(6e7 // (ny * nz)))
    for i in range(0, planes.shape[0], step):
        m = planes[i:i + step].bool()
        last = torch.where(m, at, -far).cummax(2).values
        nxt = torch.where(m, at, 2 * far).flip(2).cummin(2).values.flip(2)
        g = torch.minimum(at - last, nxt - at).square_()
        best = g.clone()
        top = float("inf")
        for d in range(1, min(ny, most)):
            if d % 16 == 1:
                top = float(best.max())
            if d * d >= top:
                break
            torch.minimum(best[:, d:], g[:, :-d] + d * d, out=best[:, d:])
            torch.minimum(best[:, :-d], g[:, d:] + d * d, out=best[:, :-d])
        out[i * ny * nz:][:best.numel()] = best.view(-1)
    return out


def grid(case, sm):
    q = f32(quats(case["n_q"], sm["rng"]))
    return q


def voxel_in(sm, n):
    """n voxels: a random grain each, near its centre."""
    g = sm["rng"].integers(0, len(sm["q"]), n)
    d = sm["rng"].normal(size=(n, 3)) * sm["size"][g][:, None] * 0.3
    return g, f32(sm["cen"][g] + d)


def euler(q):
    m = matrices(torch.tensor(q)).numpy()
    e = np.stack([np.arctan2(m[:, 0, 2], -m[:, 1, 2]), np.arccos(np.clip(m[:, 2, 2], -1, 1)),
                  np.arctan2(m[:, 2, 0], m[:, 2, 1])], 1)
    return f32(np.degrees(e) % 360)


VOX, DIM = 0.0025, 160     # voxel [mm] and side of the volume of voxel indices
PARAM1 = f32([1, 1, 1, 1, VOX, 0, 0, 0, DIM, DIM, DIM, 0.6, 0.05, 10.0])


def voxel_pos(idx):
    """Centre of 1-based voxel indices (x and y mirrored, as the volume's frame has them)."""
    p = (np.asarray(idx, np.float64) - DIM / 2) * float(PARAM1[4])
    return p * np.array([-1.0, -1.0, 1.0])


def matched(case, sm):
    """Matched spots of random grains: (grains n x 6, grain, iw, ih, uv, offsets)."""
    geo, rng = sm["geo"], sm["rng"]
    most = case.get("spots", 1 << 40)
    n = case.get("grains", most // (geo["c"].numel() * geo["h"].shape[0] // 8) + 2)
    q = quats(n, rng)
    q = q[np.argsort(-q[:, 0])]
    q[:, 0] = np.maximum(q[:, 0], 0.2)   # Rodrigues vectors of moderate length, as reduced orientations have
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    phi, rr = rng.uniform(0, 2 * np.pi, n), sm["rad"] * np.sqrt(rng.random(n))
    cen = np.stack([rr * np.cos(phi), rr * np.sin(phi), rng.uniform(-sm["rad"], sm["rad"], n)], 1)
    gr = torch.tensor(np.concatenate([q[:, 1:] / q[:, :1], cen], 1), device=DEV)
    U = matrices(torch.tensor(q, device=DEV))
    parts, step = [], per_chunk(geo)
    for i in range(0, n, step):
        ok, u, v, _ = landings(geo, gr[i:i + step, 3:], U[i:i + step])
        at = ok.nonzero()
        parts.append((at[:, 0] + i, at[:, 1], at[:, 2], torch.stack([u[ok], v[ok]], 1)))
    grain, iw, ih, uv = (torch.cat(x)[:most].contiguous() for x in zip(*parts))
    gen = torch.Generator(device=DEV).manual_seed(int(rng.integers(1 << 30)))
    uv = uv + 0.5 * torch.randn(uv.shape, dtype=torch.float64, device=DEV, generator=gen)
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.bincount(grain, minlength=n).cumsum(0)
    return gr, grain.int(), iw.int(), ih.int(), uv.reshape(-1).contiguous(), off


def room(case, geo):
    """Pairs that the caller's buffer holds: a quarter of a trial's reflections and some."""
    return case["trials"] * (case["nrot"] * len(geo["hkl"]) // 4 + 64) + 1024


def geo10_of(geo):
    P = geo["P"]
    return np.array([P["lss"], P["lsd"], 0, 0, *geo["tilt"], 0, 0, 0], np.float64)


def inputs(case, seed):
    """All inputs of a case, without the framework."""
    kind = case["kind"]
    sm = sample(case, seed, kind in ("scan", "batch", "grow", "compete", "index", "pair", "masks"))
    rng = sm["rng"]
    if kind in ("scan", "masks"):
        sm["pos"], sm["grid"] = voxel_in(sm, 1)[1][0], grid(case, sm)
    elif kind in ("batch", "index"):
        sm["grain"], sm["pos"] = voxel_in(sm, case["seeds"])
        sm["grid"] = grid(case, sm)
    elif kind == "grow":
        g = int(rng.integers(len(sm["q"])))
        c = np.round(sm["cen"][g] * [-1, -1, 1] / VOX + DIM / 2)
        r = int(np.ceil((3 * case["voxels"] / (4 * np.pi)) ** (1 / 3))) + 1
        ax = np.arange(-r, r + 1)
        d = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
        d = d[np.argsort((d ** 2).sum(1), kind="stable")][:case["voxels"]]
        m = len(d)
        sm["rows"] = f32(np.concatenate([np.clip(c + d, 1, DIM), rng.uniform(0, 0.9, (m, 1)), rng.integers(0, 8, (m, 1)) > 0,
                                         rng.choice([2.0, 20.0], (m, 1))], 1))
        sm["U"] = f32(matrices(torch.tensor(sm["q"][g:g + 1])).numpy().reshape(9))
    elif kind == "compete":
        n, m, var = len(sm["q"]), case["voxels"], 33
        g = rng.integers(0, n, m)
        idx = np.clip(np.round(sm["cen"][g] * [-1, -1, 1] / VOX + DIM / 2 + rng.normal(size=(m, 3)) * 4), 1, DIM)
        k = np.minimum(rng.geometric(0.15, m), 64)
        off = np.concatenate([[0], np.cumsum(k)])
        base = np.repeat(sm["q"], var, 0)
        jit = rng.normal(size=base.shape) * np.where(np.arange(len(base)) % var == 0, 0.0, 0.004)[:, None]
        q = base + jit
        sm["euler"] = euler(q / np.linalg.norm(q, axis=1, keepdims=True))
        own = np.where(rng.random(off[-1]) < 0.7, np.repeat(g, k), rng.integers(0, n, off[-1]))
        sm["ids"] = f32(own * var + rng.integers(0, var, off[-1]) + 1)
        sm["rows"] = f32(np.concatenate([idx, off[:-1, None] + 1, off[1:, None]], 1))
    elif kind == "pair":
        n = case["trials"]
        g, pos = voxel_in(sm, n)
        geo = sm["geo"]
        sm["tpos"] = torch.tensor(pos.astype(np.float64), device=DEV)
        sm["tq"] = torch.tensor(sm["q"][g], device=DEV)
        few = min(len(sm["q"]), 40)
        lists = []
        for i in range(0, few, per_chunk(geo)):
            ok, u, v, _ = landings(geo, torch.tensor(sm["cen"][i:min(few, i + per_chunk(geo))], device=DEV),
                                   matrices(torch.tensor(sm["q"][i:min(few, i + per_chunk(geo))], device=DEV)))
            lists.append((ok.nonzero()[:, 1], torch.stack([u[ok], v[ok]], 1)))
        iw, uv = torch.cat([a for a, _ in lists]), torch.cat([b for _, b in lists])
        nrot = case["nrot"]
        gen = torch.Generator(device=DEV).manual_seed(int(seed) + 9)
        uv = uv + 0.5 * torch.randn(uv.shape, dtype=torch.float64, device=DEV, generator=gen)
        odd = torch.rand(20 * nrot, 2, dtype=torch.float64, device=DEV, generator=gen)
        uv = torch.cat([uv, odd * torch.tensor([geo["ny"], geo["nz"]], dtype=torch.float64, device=DEV)])
        iw = torch.cat([iw, torch.arange(nrot, device=DEV).repeat(20)])
        order = torch.argsort(iw, stable=True)
        area = 4 + 36 * torch.rand(len(iw), 1, dtype=torch.float64, device=DEV, generator=gen)
        sm["spots"] = torch.cat([uv[order], area], 1).contiguous()
        sm["proj"] = torch.zeros(nrot + 1, dtype=torch.int64, device=DEV)
        sm["proj"][1:] = torch.bincount(iw, minlength=nrot).cumsum(0)
    else:
        sm["truth"], sm["grain"], sm["iw"], sm["ih"], sm["uv"], sm["off"] = matched(case, sm)
        n = len(sm["truth"])
        gen = torch.Generator(device=DEV).manual_seed(int(seed) + 5)
        if kind != "geometry":
            move = torch.randn(n, 6, dtype=torch.float64, device=DEV, generator=gen)
            sm["start"] = sm["truth"] + move * torch.tensor([0.005] * 3 + [0.003] * 3, dtype=torch.float64, device=DEV)
        else:
            px = sm["geo"]["px"]
            half = np.array([0.5, 0.5, 20 * px, 20 * px, 1, 1, 1, 0.02, 0.02, 0.02])
            sm["start"] = torch.tensor(geo10_of(sm["geo"]) + rng.uniform(-1, 1, (case["starts"], 10)) * half, device=DEV)
    return sm


# ---- what a program has in hand, and one pass -------------------------------------------------------

def prepare(case, seed):
    from grainrecon_b200 import fit, seeding
    from grainrecon_b200._lib import Context

    kind, sm = case["kind"], inputs(case, seed)
    geo = sm["geo"]
    ctx = Context(0)
    ctx.set_geometry(*geo["args"])
    st = {"case": case, "ctx": ctx, "args": geo["args"], "sm": sm}
    if kind == "masks":
        st["map"] = torch.empty(sm["mask"].numel(), dtype=torch.float32, device=DEV)
    elif "mask" in sm:
        ctx.upload_masks(distance(sm.pop("mask"), case).sqrt_(), case["nz"], case["ny"], case["nrot"])
    torch.cuda.empty_cache()
    if kind == "scan":
        ctx.set_median(case["median"])
        st["out"] = np.empty(4 * case["n_q"], np.float32)
    elif kind == "batch":
        n, N = case["seeds"], case["n_q"]
        ctx.set_median(case["median"])
        st["d_pos"], st["d_q"] = (torch.tensor(x.reshape(-1), device=DEV) for x in (sm["pos"], sm["grid"]))
        st["out"] = torch.empty(n * N * 4, dtype=torch.float32, device=DEV)
        st["best"] = torch.empty(n, dtype=torch.int32, device=DEV)
        st["best_c"] = torch.empty(n, dtype=torch.float32, device=DEV)
    elif kind == "compete":
        st["d"] = [torch.tensor(sm[k].reshape(-1), device=DEV) for k in ("rows", "ids", "euler")]
        st["out"] = torch.empty(8 * case["voxels"], dtype=torch.float32, device=DEV)
    elif kind == "index":
        st["indexer"] = seeding.SeedIndexer(ctx, sm["grid"].astype(np.float64), case["top"])
    elif kind == "pair":
        st["room"] = room(case, geo)
        st["pairs"] = torch.zeros(9 * st["room"], dtype=torch.float64, device=DEV)
        st["found"] = ctypes.c_int64()
    elif kind in ("grains", "geometry", "jacobian"):
        st["spots"] = fit.Spots(sm["grain"], sm["iw"], sm["ih"], sm["uv"], sm["off"])
        st["geo10"] = geo10_of(geo)
        st["d_truth"] = sm["truth"].reshape(-1).contiguous()
        st["d_start"] = sm["start"].reshape(-1).contiguous()
    return st


def run(st):
    case, ctx, sm = st["case"], st["ctx"], st["sm"]
    kind = case["kind"]
    S9, B9, hkl, rot, R9, par = st["args"]
    if kind == "scan":
        return ctx.forward_comp(sm["pos"], sm["grid"], S9, B9, hkl, None, rot, R9, par, out=st["out"])
    if kind == "batch":
        ctx.forward_comp_argmax_device(st["d_pos"], case["seeds"], st["d_q"], case["n_q"], st["out"], st["best"],
                                       st["best_c"])
        return {"out": st["out"], "best": st["best"], "best_c": st["best_c"]}
    if kind == "grow":
        return ctx.grow_indexed_region(sm["rows"], sm["U"], S9, B9, hkl, None, rot, R9, par, PARAM1)
    if kind == "compete":
        rows, ids, eu = st["d"]
        ctx.compete_device(rows, case["voxels"], ids, ids.numel(), eu, eu.numel() // 3, PARAM1, st["out"])
        return st["out"]
    if kind == "index":
        rows, cand = st["indexer"].index(np.arange(1, case["seeds"] + 1), sm["pos"].astype(np.float64))
        return {"rows": rows, "cand": cand}
    if kind == "pair":
        torch.cuda.current_stream().synchronize()   # the inputs, before the library's own stream reads them
        ctx._check(ctx.L.grc_pair_spots(ctx.h, sm["tpos"].data_ptr(), sm["tq"].data_ptr(), case["trials"],
                                        sm["spots"].data_ptr(), len(sm["spots"]), sm["proj"].data_ptr(),
                                        st["pairs"].data_ptr(), st["room"], ctypes.byref(st["found"])))
        rec = st["pairs"].view(-1, 9)
        return {"found": st["found"].value, "which": rec.view(torch.int32)[:, :4], "values": rec[:, 2:]}
    if kind == "masks":
        ny, nz, nrot = case["ny"], case["nz"], case["nrot"]
        ctx.edt(sm["mask"], nz, ny, nrot, st["map"])
        ctx.upload_masks(st["map"], nz, ny, nrot)
        out = ctx.forward_comp(sm["pos"], sm["grid"], S9, B9, hkl, None, rot, R9, par)
        return {"map": st["map"], "distinct": ctx.mask_info()["n_distinct"], "scan": out}
    from grainrecon_b200 import fit

    if kind == "jacobian":
        res, jac = fit.residual_jacobian(ctx, case["mode"], st["geo10"], st["d_start"], st["spots"])
        return {"res": res, "jac": jac}
    n = st["d_start"].numel() // (6 if kind == "grains" else 10)
    d, lam = st["d_start"].clone(), torch.full((n,), 1e-3, dtype=torch.float64, device=DEV)
    if kind == "grains":
        got = fit.grains_lm(ctx, st["geo10"], d, st["spots"], lam, case["iters"])
    else:
        got = fit.geometry_lm(ctx, d, st["d_truth"], st["spots"], lam, 1)
    return {"params": d, "lambda": lam, "improved": got}


# ---- the results in 64 bits -------------------------------------------------------------------------

def columns(geo, dmap, pos, U, median=True):
    """[Nr_simu Nr_intersect completeness dis_median] of trials (pos n x 3, U n x 3 x 3)."""
    rows, step = [], per_chunk(geo)
    for i in range(0, len(pos), step):
        ok, u, v, _ = landings(geo, pos[i:i + step], U[i:i + step])
        dis = torch.full(ok.shape, float("inf"), dtype=torch.float32, device=DEV)
        dis[ok] = dmap[pixel(geo, ok, u, v)]
        n = ok.flatten(1).sum(1)
        r = [n, ((dis <= HIT) & ok).flatten(1).sum(1)]
        if median:
            d = dis.flatten(1).sort(1).values
            lo, hi = ((n - 1) // 2).clamp(min=0), (n // 2).clamp(max=d.shape[1] - 1)
            med = (d.gather(1, lo[:, None])[:, 0].double() + d.gather(1, hi[:, None])[:, 0].double()) / 2
            r.append(torch.where(n > 0, med, 2000.0))
        else:
            r.append(torch.full_like(n, float("nan"), dtype=torch.float64))
        rows.append(torch.stack([r[0].double(), r[1].double(), r[1].double() / r[0].double(), r[2]], 1))
    return torch.cat(rows)


def spot_uv(geo, e, gr, sm, lo=0, hi=None):
    """(u, v) of matched spots: e = 10 geometry tensors or numbers, gr = 6 grain tensors per spot."""
    hi = len(sm["iw"]) if hi is None else hi
    rr = gr[0] ** 2 + gr[1] ** 2 + gr[2] ** 2
    a = 1 / torch.sqrt(1 + rr)
    U = matrices(torch.stack([a, gr[0] * a, gr[1] * a, gr[2] * a], -1))
    h = geo["h"][sm["ih"][lo:hi].long()].to(U.dtype)
    g = torch.einsum("nij,nj->in", U, h)
    iw = sm["iw"][lo:hi].long()
    P = {"lss": e[0], "lsd": e[1], "y00": e[2], "z00": e[3], "R": rot_det(e[4], e[5], e[6]), "p0y": e[7], "p0z": e[8],
         "rao": e[9]}
    u, v, _, _ = land(P, gr[3:], g, geo["c"][iw], geo["s"][iw], geo)
    return u, v


def derivatives(geo, e, gr, sm, mode, lo=0, hi=None):
    """(u, v, du, dv) of matched spots by complex steps over the 6 grain or 10 geometry parameters."""
    du, dv, step = [], [], 1e-30
    hi = len(sm["iw"]) if hi is None else hi
    base = gr[sm["grain"][lo:hi].long()].t()
    for k in range(6 if mode == 0 else 10):
        ek = [torch.tensor(complex(float(x), step if mode == 1 and i == k else 0.0), dtype=torch.complex128, device=DEV)
              for i, x in enumerate(e)]
        gk = [x.to(torch.complex128) + (1j * step if mode == 0 and i == k else 0.0) for i, x in enumerate(base)]
        u, v = spot_uv(geo, ek, gk, sm, lo, hi)
        du.append(u.imag / step)
        dv.append(v.imag / step)
    return u.real, v.real, torch.stack(du, 1), torch.stack(dv, 1)


def normal(geo, e, gr, sm, mode):
    """J'J, J'r per grain (mode 0) or in all (mode 1)."""
    k, n = (6, len(gr)) if mode == 0 else (10, 1)
    A = torch.zeros(n, k, k, dtype=torch.float64, device=DEV)
    b = torch.zeros(n, k, dtype=torch.float64, device=DEV)
    uv = sm["uv"].view(-1, 2)
    for lo in range(0, len(uv), 1 << 21):
        hi = min(len(uv), lo + (1 << 21))
        u, v, du, dv = derivatives(geo, e, gr, sm, mode, lo, hi)
        ru, rv = u - uv[lo:hi, 0], v - uv[lo:hi, 1]
        if mode == 1:
            A[0] += du.t() @ du + dv.t() @ dv
            b[0] += du.t() @ ru + dv.t() @ rv
        else:
            g = sm["grain"][lo:hi].long()
            A.index_add_(0, g, du[:, :, None] * du[:, None] + dv[:, :, None] * dv[:, None])
            b.index_add_(0, g, du * ru[:, None] + dv * rv[:, None])
    return A, b


def cost(geo, e, gr, sm, mode):
    uv = sm["uv"].view(-1, 2)
    e = [torch.tensor(float(x), dtype=torch.float64, device=DEV) for x in e]
    g = sm["grain"].long()
    u, v = spot_uv(geo, e, list(gr[g].t()), sm)
    r = (u - uv[:, 0]) ** 2 + (v - uv[:, 1]) ** 2
    return r.sum() if mode == 1 else torch.zeros(len(gr), dtype=torch.float64, device=DEV).index_add_(0, g, r)


def damped(A, b, lam):
    """(A + lam diag A) x = -b; no step where A is not positive definite."""
    M = A + lam[:, None, None] * torch.diag_embed(torch.diagonal(A, dim1=1, dim2=2))
    L, info = torch.linalg.cholesky_ex(M)
    x = torch.cholesky_solve(-b[:, :, None], L)[:, :, 0]
    return torch.where((info == 0)[:, None], x, 0.0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "index":
        return None        # the path of a discrete search: no value of its own in more bits
    if kind == "batch" and case["seeds"] * case["n_q"] * case["nrot"] > 1e8:
        return None        # minutes
    sm = inputs(case, seed)
    geo = sm["geo"]
    if kind in ("grains", "geometry", "jacobian"):
        return exact_fit(case, sm, geo)
    dmap = distance(sm["mask"], case, 1 << 30 if kind == "masks" else 96).sqrt_()
    if kind in ("scan", "masks"):
        U = matrices(torch.tensor(sm["grid"].astype(np.float64), device=DEV))
        pos = torch.tensor(sm["pos"].astype(np.float64), device=DEV).expand(len(U), 3)
        out = columns(geo, dmap, pos, U, case.get("median", True)).reshape(-1)
        return out if kind == "scan" else {"map": distance(sm["mask"], case, 1 << 30).double().sqrt_(), "distinct": None,
                                           "scan": out}
    if kind == "batch":
        N = case["n_q"]
        U = matrices(torch.tensor(sm["grid"].astype(np.float64), device=DEV))
        out = torch.cat([columns(geo, dmap, torch.tensor(p.astype(np.float64), device=DEV).expand(N, 3), U,
                                 case["median"]) for p in sm["pos"]])
        c = out[:, 2].view(-1, N)
        return {"out": out.reshape(-1), "best": None, "best_c": torch.where(c.isnan(), -1.0, c).max(1).values}
    if kind == "grow":
        rows = sm["rows"].astype(np.float64)
        pos = torch.tensor(voxel_pos(rows[:, :3]), device=DEV)
        U = torch.tensor(sm["U"].astype(np.float64).reshape(1, 3, 3), device=DEV).expand(len(rows), 3, 3)
        c = columns(geo, dmap, pos, U)
        r = torch.tensor(rows, device=DEV)
        p1 = PARAM1.astype(np.float64)
        flag = (r[:, 4] > 0) & (c[:, 2] > r[:, 3]) & (c[:, 3] <= r[:, 5].clamp(max=p1[13])) & (
            c[:, 2] >= p1[11] * (1 - p1[12]))
        return torch.cat([r[:, :3], c[:, :2], c[:, 3:], flag[:, None].double()], 1).reshape(-1)
    if kind == "compete":
        rows = sm["rows"].astype(np.int64)
        k = rows[:, 4] - rows[:, 3] + 1
        e = torch.tensor(sm["euler"].astype(np.float64), device=DEV) * math.pi / 180
        c1, c, c2 = torch.cos(e).unbind(1)
        s1, s, s2 = torch.sin(e).unbind(1)
        U = torch.stack([c1 * c2 - s1 * s2 * c, -c1 * s2 - s1 * c2 * c, s1 * s, s1 * c2 + c1 * s2 * c,
                         -s1 * s2 + c1 * c2 * c, -c1 * s, s2 * s, c2 * s, c], 1).view(-1, 3, 3)
        pos = torch.tensor(voxel_pos(rows[:, :3]), device=DEV)
        ids = torch.tensor(sm["ids"], device=DEV).long() - 1
        own = torch.repeat_interleave(torch.arange(len(rows), device=DEV), torch.tensor(k, device=DEV))
        c = columns(geo, dmap, pos[own], U[ids])
        C = torch.where(c[:, 2].isnan(), -1.0, c[:, 2])
        best = torch.full((len(rows),), -2.0, dtype=torch.float64, device=DEV).scatter_reduce_(0, own, C, "amax")
        at = torch.where(C == best[own], torch.arange(len(own), device=DEV), len(own))
        first = torch.full((len(rows),), len(own), device=DEV).scatter_reduce_(0, own, at, "amin")
        ed = torch.tensor(sm["euler"].astype(np.float64), device=DEV)[ids[first]]
        return torch.cat([torch.arange(1, len(rows) + 1, device=DEV)[:, None].double(), ed,
                          (ids[first] + 1)[:, None].double(), c[first][:, 2:3], c[first][:, 1:2], c[first][:, 3:]],
                         1).reshape(-1)
    return exact_pairs(case, sm, geo, dmap)


def exact_pairs(case, sm, geo, dmap):
    """Every hit's nearest centroid of its projection, when near enough, in (trial, projection, reflection) order."""
    got, step = [], max(1, per_chunk(geo) // 4)
    off = sm["proj"].tolist()
    most = max(b - a for a, b in zip(off, off[1:]))
    pad = torch.full((case["nrot"], most, 3), 1e9, dtype=torch.float64, device=DEV)
    for i, (a, b) in enumerate(zip(off, off[1:])):
        pad[i, :b - a] = sm["spots"][a:b]
    for i in range(0, case["trials"], step):
        ok, u, v, lam = landings(geo, sm["tpos"][i:i + step], matrices(sm["tq"][i:i + step]))
        dis = dmap[pixel(geo, ok, u, v)].double()
        at, y, z = ok.nonzero()[:, 1], torch.floor(u[ok] + 0.5), torch.floor(v[ok] + 0.5)
        hit = dis <= HIT
        at, y, z, en, dis = at[hit], y[hit], z[hit], 12.398 / lam[ok][hit], dis[hit]
        near = []
        for j in range(0, len(at), 1 << 18):
            s = pad[at[j:j + (1 << 18)]]
            d = torch.sqrt((s[:, :, 0] - y[j:j + (1 << 18), None]) ** 2 + (s[:, :, 1] - z[j:j + (1 << 18), None]) ** 2)
            m, k = d.min(1)
            near.append(torch.cat([m[:, None], s.gather(1, k[:, None, None].expand(-1, 1, 3))[:, 0]], 1))
        if near:
            near = torch.cat(near)
            keep = near[:, 0] < torch.sqrt(near[:, 3]).clamp(max=15.0)
            got.append(torch.cat([y[:, None], z[:, None], near[:, 1:], en[:, None], dis[:, None]], 1)[keep])
    out = torch.zeros(room(case, geo), 7, dtype=torch.float64, device=DEV)
    if got:
        got = torch.cat(got)
        out[:len(got)] = got
    return {"found": None, "which": None, "values": out}


def exact_fit(case, sm, geo):
    kind = case["kind"]
    uv = sm["uv"].view(-1, 2)
    if kind == "jacobian":
        parts = []
        for lo in range(0, len(uv), 1 << 20):
            hi = min(len(uv), lo + (1 << 20))
            u, v, du, dv = derivatives(geo, geo10_of(geo), sm["start"], sm, case["mode"], lo, hi)
            parts.append((torch.stack([u, v], 1) - uv[lo:hi], torch.stack([du, dv], 1)))
        return {"res": torch.cat([p[0] for p in parts]), "jac": torch.cat([p[1] for p in parts])}
    mode = 0 if kind == "grains" else 1
    x = sm["start"].clone()
    lam = torch.full((len(x),), 1e-3, dtype=torch.float64, device=DEV)
    for _ in range(case.get("iters", 1)):
        if mode == 0:
            e = geo10_of(geo)
            new = x + damped(*normal(geo, e, x, sm, 0), lam)
            now, then = cost(geo, e, x, sm, 0), cost(geo, e, new, sm, 0)
        else:
            Ab = [normal(geo, e.tolist(), sm["truth"], sm, 1) for e in x]
            new = x + damped(torch.cat([a for a, _ in Ab]), torch.cat([b for _, b in Ab]), lam)
            now, then = (torch.stack([cost(geo, e.tolist(), sm["truth"], sm, 1) for e in y]) for y in (x, new))
        better = then < now
        x = torch.where(better[:, None], new, x)
        lam = torch.where(better, (lam * 0.1).clamp(min=1e-9), (lam * 10).clamp(max=1e9))
    return {"params": x.reshape(-1), "lambda": lam, "improved": None}


# ---- what one pass cannot do without -----------------------------------------------------------------

CHAIN = 130                # operations of one landing
SHARE = 0.2                # of the (projection, reflection) pairs that fall into the energy window


def work(case):
    kind = case["kind"]
    nh = 86 if case["lattice"] == "fe" else 64
    pairs = case["nrot"] * nh
    pixels = case["nrot"] * case["ny"] * case["nz"]
    per_trial = pairs * (5 + SHARE * CHAIN)
    if kind in ("scan", "batch"):
        n, seeds = case["n_q"], case.get("seeds", 1)
        reads = min(pixels / 8 if not case["median"] else pixels, n * seeds * pairs * SHARE * 32)
        return {"bytes": 16.0 * n + 16.0 * n * seeds + reads, "flops": float(n) * seeds * per_trial}
    if kind in ("grow", "compete"):
        n = case["voxels"] * (1 if kind == "grow" else 6.6)
        return {"bytes": 60.0 * case["voxels"] + min(pixels, n * pairs * SHARE * 32), "flops": n * per_trial}
    if kind == "index":
        n = case["seeds"] * (case["n_q"] + 730 * min(case["top"], case["n_q"]))
        return {"bytes": 16.0 * n + min(pixels / 8, n * pairs * SHARE * 32), "flops": n * per_trial}
    if kind == "pair":
        return {"bytes": case["trials"] * pairs * SHARE * (32 + 72), "flops": case["trials"] * per_trial}
    if kind == "masks":
        return {"bytes": pixels * (1 + 4 + 4 + 2 + 1), "flops": pixels * 4.0}
    spots = case.get("spots", case.get("grains", 0) * pairs * SHARE)
    if kind == "grains":
        return {"bytes": 28.0 * spots, "flops": spots * case["iters"] * (2 * CHAIN + 6 * 2 * CHAIN)}
    if kind == "geometry":
        return {"bytes": 28.0 * spots, "flops": spots * case["starts"] * (2 * CHAIN + 10 * 2 * CHAIN)}
    k = 6 if case["mode"] == 0 else 10
    return {"bytes": spots * (28 + 16 * (1 + k)), "flops": spots * CHAIN * (1 + k)}

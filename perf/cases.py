"""The work a user of range_libc_gb300 has it do, as measurable cases.

A case is a dict of plain values.  ``prepare`` builds what a user's program holds before the call
(map, method, sensor table, arrays), ``run`` makes one pass through the public entry points with
the schedules a caller gets without asking for others, ``work`` states the bytes and operations
the pass cannot do without, and ``exact`` recomputes its numbers in 64 bits with plain torch.

Sizes are the repository's own workloads (512^2 and 2048^2 maps, 4,000 x 61 particle-filter steps,
10,000 and 1,000,000 queries, theta discretisations 108 and 216, 500-20,000 particles x 30-1,081
beams, max_range 100-400 px, 65,536-ray training batches) and odd ones between them.
"""
import math

import numpy as np
import torch

from range_libc_gb300 import range_libc as rl
from range_libc_gb300 import workloads as W

M_2PI = 6.28318530718
ROS_SCALE = 0.05                      # m per cell of the corridor maps, as a ROS map server gives them
IDENTITY = (1.0, 0.0, 0.0, 0.0, 0.0, 1.0)
DEV = "cuda:0"
PARAMS = 328961                       # of the learned surrogate: 512 -> 4 x 256 -> 1


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a simulator's or planner's single lidar scan: one pose, 1,081 beams, numpy buffers -- the
        # smallest call, all launch and latency
        {"name": "scan_rm_1x1081_host", "family": "scan", "kind": "rm", "side": 2048, "poses": 1, "beams": 1081,
         "max_range": 200.0},
        # the particle-filter step of a robot: 4,000 particles x 61 beams, numpy buffers, fused call
        {"name": "pf_rm_4000x61_host", "family": "pf", "kind": "rm", "side": 2048, "particles": 4000, "beams": 61,
         "max_range": 200.0, "device": False, "td": 0},
        # a large filter on a full 1,081-beam lidar, arrays resident on the GPU
        {"name": "pf_rm_20000x1081_dev", "family": "pf", "kind": "rm", "side": 2048, "particles": 20000,
         "beams": 1081, "max_range": 200.0, "device": True, "td": 0},
        # the unfused step that callers written for the CPU library use: ranges, then the sensor model
        {"name": "plain_cddt_4000x108_dev", "family": "plain", "kind": "cddt", "side": 2048, "particles": 4000,
         "beams": 108, "max_range": 200.0, "device": True, "td": 108},
        # independent queries, Bresenham's line on a small map, numpy buffers
        {"name": "many_bl_10k_host", "family": "many", "kind": "bl", "side": 512, "queries": 10000,
         "max_range": 300.0, "device": False, "td": 0},
        # independent ray-marching queries all over a map (the reference's random-sample benchmark)
        {"name": "many_rm_2M_dev", "family": "many", "kind": "rm", "side": 2048, "queries": 2000000,
         "max_range": 300.0, "device": True, "td": 0},
        # the same of the compressed table
        {"name": "many_cddt_1M_dev", "family": "many", "kind": "cddt", "side": 2048, "queries": 1000000,
         "max_range": 300.0, "device": True, "td": 108},
        # and of the full lookup table
        {"name": "many_glt_1M_dev", "family": "many", "kind": "glt", "side": 2048, "queries": 1000000,
         "max_range": 300.0, "device": True, "td": 108},
        # many robots' filters, uneven in maps, particles, beams and ranges, in one launch
        {"name": "batch_8_filters", "family": "batch", "filters": 8, "spec_seed": 4000, "most_side": 4096},
        # a map arrives (or changed): build its ray marcher and cast the first step's rays
        {"name": "setup_rm_2048", "family": "setup", "kind": "rm", "side": 2048, "particles": 4000, "beams": 61,
         "max_range": 200.0, "td": 0},
        # the learned surrogate: 10,000 poses x 108 beams predicted, checked, recast where rejected
        {"name": "learned_query_10000x108", "family": "learned_query", "side": 2048, "particles": 10000,
         "beams": 108, "max_range": 300.0},
        # and its training: rays drawn by the marcher, forward, backward, Adam
        {"name": "learned_train_65536", "family": "learned_train", "side": 1024, "batch": 65536, "steps": 2,
         "max_range": 300.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; its rays are at most those of the largest listed case."""
    family = rng.choice(["scan", "pf", "pf", "plain", "many", "many", "many", "batch", "setup", "learned_query",
                         "learned_train"])
    side = rng.choice([512, 777, 1024, 1500, 2048])
    max_range = round(rng.uniform(100.0, 400.0), 1)
    if family == "scan":
        return {"family": family, "kind": rng.choice(["rm", "bl", "cddt"]), "side": side, "poses": rng.randint(1, 16),
                "beams": rng.randint(30, 1081), "max_range": max_range}
    if family in ("pf", "plain"):
        kind = rng.choice(["rm", "rm", "bl", "cddt"])
        return {"family": family, "kind": kind, "side": side, "particles": _log_int(rng, 500, 8000),
                "beams": _log_int(rng, 30, 1081), "max_range": max_range, "device": rng.random() < 0.5,
                "td": rng.choice([108, 216]) if kind == "cddt" else 0}
    if family == "many":
        kind = rng.choice(["rm", "bl", "cddt", "pcddt", "glt"])
        return {"family": family, "kind": kind, "side": side, "queries": _log_int(rng, 10000, 1000000),
                "max_range": max_range, "device": rng.random() < 0.75,
                "td": rng.choice([107, 108, 216]) if kind in ("cddt", "pcddt") else (108 if kind == "glt" else 0)}
    if family == "batch":
        return {"family": family, "filters": rng.randint(2, 6), "spec_seed": rng.randint(1, 10 ** 6), "most_side": 2048}
    if family == "setup":
        kind = rng.choice(["rm", "cddt", "glt"])
        return {"family": family, "kind": kind, "side": rng.choice([400, 512, 1024, 1500, 2048]),
                "particles": _log_int(rng, 500, 4000), "beams": rng.randint(30, 108), "max_range": max_range,
                "td": 0 if kind == "rm" else 108}
    if family == "learned_query":
        return {"family": family, "side": side, "particles": _log_int(rng, 100, 10000), "beams": rng.randint(30, 108),
                "max_range": max_range}
    return {"family": "learned_train", "side": rng.choice([512, 1024]), "batch": 128 * _log_int(rng, 32, 512),
            "steps": rng.randint(1, 2), "max_range": max_range}


# ------------------------------------------------------------------ inputs
def _corridor_inputs(case, seed):
    """A corridor map at ROS_SCALE, poses about a free point, beams over 270 degrees, a tempered
    sensor table (the likelihood to the power 30 / beams, so that the product over correlated beams
    stays a usable weight) and an observed scan."""
    rng = np.random.default_rng(seed)
    occ = W.corridor_map(case["side"], seed % 1000003)
    n, na, mr = case.get("particles", case.get("poses")), case["beams"], case["max_range"]
    while True:
        gx, gy = rng.uniform(60, case["side"] - 60, 2)
        if not occ[int(gx) - 4:int(gx) + 5, int(gy) - 4:int(gy) + 5].any():
            break
    world = (ROS_SCALE, 0.0, -12.5, -7.5, 0.0, 1.0)
    head = rng.uniform(0, 2 * math.pi)
    first = 1 if "poses" in case else 0          # a scan's first pose is the true one
    px, py, th = rng.normal(gx, 20.0, n), rng.normal(gy, 20.0, n), rng.normal(head, 0.3, n)
    px[:first], py[:first], th[:first] = gx, gy, head
    xw, yw = W.grid_to_world(px, py, world)
    ins = np.stack([xw, yw, th], 1).astype(np.float32)
    angles = W.laser_angles(na)
    K = int(mr) + 1
    table = W.sensor_table(K) ** min(1.0, 30.0 / na)
    t = np.arange(0.0, mr, 0.5)
    dirs = -head - 1.5 * math.pi - angles.astype(np.float64)
    cx = np.clip((gx + np.cos(dirs)[:, None] * t).astype(int), 0, case["side"] - 1)
    cy = np.clip((gy + np.sin(dirs)[:, None] * t).astype(int), 0, case["side"] - 1)
    hit = occ[cx, cy] != 0
    seen = np.where(hit.any(1), t[hit.argmax(1)], mr) + rng.normal(0, 2.0, na)
    return {"occ": occ, "world": world, "ins": ins, "angles": angles, "table": table,
            "obs": (seen * ROS_SCALE).astype(np.float32)}


def _free_poses(occ, n, rng):
    """n poses uniform over free cells, swapped for the world API's axis order, any heading."""
    free = np.flatnonzero(occ.reshape(-1) == 0)
    pick = free[rng.integers(0, len(free), n)]
    q = np.empty((n, 3), np.float32)
    q[:, 1] = (pick // occ.shape[1]) + rng.random(n)
    q[:, 0] = (pick % occ.shape[1]) + rng.random(n)
    q[:, 2] = rng.uniform(0.0, 2.0 * math.pi, n)
    return q


def _spread_inputs(case, seed):
    """A rectangles-and-disks map in grid units and poses all over its free cells."""
    rng = np.random.default_rng(seed)
    occ = W.rect_disk_map(case["side"], seed % 1000003)
    d = {"occ": occ, "world": IDENTITY, "ins": _free_poses(occ, case.get("queries", case.get("particles", 0)), rng)}
    if "beams" in case:
        d["angles"] = W.laser_angles(case["beams"])
    return d


def _specs(case):
    """The filters of a batch: the repository's uneven ones, no map larger than most_side."""
    specs = W.uneven_batch_specs(case["filters"], case["spec_seed"])
    for s in specs:
        s.side = min(s.side, case["most_side"])
    return specs


def _filter_inputs(spec, seed):
    rng = np.random.default_rng((seed, spec.seed))
    occ = W.rect_disk_map(spec.side, (seed + spec.seed) % 1000003)
    K = int(spec.max_range) + 1
    return {"occ": occ, "world": IDENTITY, "ins": _free_poses(occ, spec.n_particles, rng),
            "angles": W.laser_angles(spec.n_beams), "table": W.sensor_table(K) ** min(1.0, 30.0 / spec.n_beams),
            "obs": rng.uniform(0, spec.max_range, spec.n_beams).astype(np.float32)}


def _inputs(case, seed):
    if case["family"] in ("scan", "pf", "plain", "setup"):
        return _corridor_inputs(case, seed)
    return _spread_inputs(case, seed)


# ------------------------------------------------------------------ state and pass
def _method(kind, omap, max_range, td):
    if kind == "rm":
        return rl.PyRayMarchingGPU(omap, max_range)
    if kind == "bl":
        return rl.PyBresenhamsLine(omap, max_range)
    if kind == "glt":
        return rl.PyGiantLUTCast(omap, max_range, td)
    m = rl.PyCDDTCast(omap, max_range, td or 108)
    if kind == "pcddt":
        m.prune()
    return m


def _omap(d):
    omap = rl.PyOMap(np.ascontiguousarray(d["occ"].T))
    omap.set_world(*d["world"][:4])
    return omap


def _on(device, a):
    return torch.from_numpy(a).to(DEV) if device else a


def _room(device, n, dtype):
    return torch.zeros(n, dtype=getattr(torch, dtype), device=DEV) if device else np.zeros(n, dtype)


def prepare(case, seed):
    f = case["family"]
    if f == "batch":
        keep, filters = [], []
        for spec in _specs(case):
            d = _filter_inputs(spec, seed)
            omap = _omap(d)
            m = rl.PyRayMarchingGPU(omap, spec.max_range)
            m.set_sensor_model(d["table"])
            filters.append((m, _on(True, d["ins"]), _on(True, d["angles"]), _on(True, d["obs"]),
                            _room(True, spec.n_particles, "float64")))
            keep.append(omap)
        return {"family": f, "batch": rl.PyFilterBatch(filters), "weights": [x[4] for x in filters], "keep": keep}
    if f == "learned_train":
        d = _spread_inputs(case, seed)
        m = rl.PyRayMarchingGPU(_omap(d), case["max_range"])
        return {"family": f, "learned": rl.PyLearnedRM(m, seed=seed % 65521), "case": case, "seed": seed % 65521}
    d = _inputs(case, seed)
    if f == "setup":
        return {"family": f, "case": case, "rows": np.ascontiguousarray(d["occ"].T != 0), "world": d["world"],
                "ins": _on(True, d["ins"]), "angles": _on(True, d["angles"]),
                "outs": _room(True, len(d["ins"]) * len(d["angles"]), "float32")}
    omap = _omap(d)
    dev = case.get("device", f == "learned_query")
    m = _method(case.get("kind", "rm"), omap, case["max_range"], case.get("td", 0))
    s = {"family": f, "method": m, "ins": _on(dev, d["ins"])}
    n = len(d["ins"])
    if f == "many":
        s["outs"] = _room(dev, n, "float32")
        return s
    s["angles"] = _on(dev, d["angles"])
    na = len(d["angles"])
    if f in ("scan", "plain", "learned_query"):
        s["outs"] = _room(dev, n * na, "float32")
    if f in ("pf", "plain"):
        m.set_sensor_model(d["table"])
        s["obs"] = _on(dev, d["obs"])
        s["weights"] = _room(dev, n, "float64")
    if f == "learned_query":
        s["learned"] = rl.PyLearnedRM(m, seed=seed % 65521)
        s["accepted"] = _room(dev, n * na, "uint8")
    return s


def run(state):
    s, f = state, state["family"]
    if f == "scan":
        s["method"].calc_range_repeat_angles(s["ins"], s["angles"], s["outs"])
        return s["outs"]
    if f == "pf":
        s["method"].calc_range_repeat_angles_eval_sensor_model(s["ins"], s["angles"], s["obs"], s["weights"])
        return s["weights"]
    if f == "plain":
        m, n, na = s["method"], len(s["ins"]), len(s["angles"])
        m.calc_range_repeat_angles(s["ins"], s["angles"], s["outs"])
        m.eval_sensor_model(s["obs"], s["outs"], s["weights"], na, n)
        return {"ranges": s["outs"], "weights": s["weights"]}
    if f == "many":
        s["method"].calc_range_many(s["ins"], s["outs"])
        return s["outs"]
    if f == "batch":
        s["batch"].run()
        return s["weights"]
    if f == "setup":
        c = s["case"]
        omap = rl.PyOMap(s["rows"])
        omap.set_world(*s["world"][:4])
        m = _method(c["kind"], omap, c["max_range"], c["td"])
        m.calc_range_repeat_angles(s["ins"], s["angles"], s["outs"])
        return s["outs"]
    if f == "learned_query":
        recast = s["learned"].calc_range_repeat_angles(s["ins"], s["angles"], s["outs"], s["accepted"])
        return {"ranges": s["outs"], "accepted": s["accepted"], "recast": recast}
    c = s["case"]
    loss = s["learned"].train(c["steps"], batch=c["batch"], lr=1e-3, seed=s["seed"])
    return {"loss": loss, "params": s["learned"].params()}


# ------------------------------------------------------------------ what a pass cannot do without
def _ray_work(kind, side, rays, max_range, td, clustered):
    """Reads of the method's table and arithmetic of `rays` casts: a march or a walk reads the part
    of the map its rays reach once (a float per cell, a bit for Bresenham's line); a table query
    reads its bin's ends and the two zero points beside it, or one 16-bit entry."""
    cells = float(min(side, 2 * (max_range + 60)) ** 2 if clustered else side * side)
    if kind == "rm":
        return min(cells, 8.0 * rays) * 4, rays * 130.0
    if kind == "bl":
        return cells / 8, rays * max_range * 6.0
    if kind == "glt":
        return rays * 2.0, rays * 20.0
    return min(rays * 16.0, 12.0 * side * side * td / 108.0), rays * 60.0


def work(case):
    f = case["family"]
    mr = case.get("max_range", 0.0)
    if f == "batch":
        b = o = 0.0
        for s in _specs(case):
            rays = float(s.n_particles) * s.n_beams
            tb, to = _ray_work("rm", s.side, rays, s.max_range, 0, False)
            b += tb + s.n_particles * 20.0 + 8.0 * (s.n_beams + (int(s.max_range) + 1) ** 2)
            o += to + rays
        return {"bytes": b, "flops": o}
    if f == "learned_train":
        rays = float(case["batch"]) * case["steps"]
        params = float(PARAMS)
        return {"bytes": case["steps"] * params * 28 + case["side"] ** 2 * 4.0,
                "flops": rays * (3 * 2 * params + 130)}
    n, na = case.get("particles", case.get("poses", case.get("queries"))), case.get("beams", 1)
    rays = float(n) * na
    b, o = _ray_work(case.get("kind", "rm"), case["side"], rays, mr, case.get("td") or 108, f not in ("many", "learned_query"))
    b += n * 12.0 + na * 4.0
    if f in ("scan", "many", "plain", "setup", "learned_query"):
        b += rays * 4.0
    if f in ("pf", "plain"):
        b += n * 8.0 + na * 4.0 + 8.0 * (int(mr) + 1) ** 2
        o += rays
    if f == "plain":
        b += rays * 4.0
    if f == "setup":          # the occupancy read, and the table written once
        cells = float(case["side"]) ** 2
        b += cells + {"rm": 4.0, "cddt": 12.0, "glt": 2.0 * case["td"]}[case["kind"]] * cells
        o += cells * (case["td"] * 130.0 if case["kind"] == "glt" else 20.0)
    if f == "learned_query":
        b += rays + PARAMS * 2.0
        o += rays * 2.0 * PARAMS
    return {"bytes": b, "flops": o}


# ------------------------------------------------------------------ 64-bit values
def _edt64(occ):
    """Distance to the nearest occupied cell, float64 [W, H] (one pass along each axis)."""
    o = torch.from_numpy(occ != 0).to(DEV)
    W_, H_ = o.shape
    far = 4 * (W_ + H_)
    y = torch.arange(H_, device=DEV).expand(W_, H_)
    before = torch.cummax(torch.where(o, y, -far), 1).values
    after = torch.flip(torch.cummin(torch.flip(torch.where(o, y, far), [1]), 1).values, [1])
    g = torch.minimum(y - before, after - y) ** 2
    best = g.clone()
    d = 1
    while d < W_ and d * d < int(best.max()):
        for e in range(d, min(d + 16, W_)):
            best[e:] = torch.minimum(best[e:], g[:-e] + e * e)
            best[:-e] = torch.minimum(best[:-e], g[e:] + e * e)
        d += 16
    return best.double().sqrt()


def _grid_rays(ins, angles, world):
    """Grid-frame (x, y, heading) of every world-frame ray, particle-major, float64."""
    s, a, ox, oy, sa, ca = world
    p = torch.from_numpy(ins).to(DEV).double()
    x, y = (p[:, 0] - ox) / s, (p[:, 1] - oy) / s
    x, y = ca * x - sa * y, sa * x + ca * y
    th = -p[:, 2] - a - 1.5 * math.pi
    if angles is not None:
        ang = torch.from_numpy(angles).to(DEV).double()
        th = (th[:, None] - ang).reshape(-1)
        x, y = x.repeat_interleave(len(ang)), y.repeat_interleave(len(ang))
    return y, x, th     # the transform hands calc_range its coordinates swapped


def _march64(dt, x, y, c, s, mr):
    out = torch.full_like(x, mr)
    live = torch.arange(len(x), device=DEV)
    t = torch.zeros_like(x)
    W_, H_ = dt.shape
    while len(live):
        px, py = torch.trunc(x + c * t).long(), torch.trunc(y + s * t).long()
        inside = (px >= 0) & (px < W_) & (py >= 0) & (py < H_)
        d = dt.reshape(-1)[torch.where(inside, px * H_ + py, 0)]
        hit = inside & (d <= 0)
        out[live[hit]] = torch.sqrt((px - x) ** 2 + (py - y) ** 2)[hit]
        t = t + torch.clamp(d * 0.999, min=1.0)
        go = inside & ~hit & (t < mr)
        live, x, y, c, s, t = live[go], x[go], y[go], c[go], s[go], t[go]
    return out


def _walk64(occ, x, y, c, s, mr):
    """Bresenham's line with the reference's float start (no rounding to cell centres)."""
    o = torch.from_numpy(occ != 0).to(DEV)
    W_, H_ = o.shape

    def occupied(gx, gy):
        inside = (gx >= 0) & (gx < W_) & (gy >= 0) & (gy < H_)
        return inside & o.reshape(-1)[torch.where(inside, torch.trunc(gx).long() * H_ + torch.trunc(gy).long(), 0)]

    out = torch.where(occupied(x, y), 0.0, mr).double()
    x1, y1 = x + mr * c, y + mr * s
    steep = (x1 - x).abs() > (y1 - y).abs()          # the walk goes along x
    u, v = torch.where(steep, x, y), torch.where(steep, y, x)
    du, dv = torch.where(steep, x1 - x, y1 - y), torch.where(steep, y1 - y, x1 - x)
    us, vs = torch.where(du > 0, 1.0, -1.0), torch.where(dv > 0, 1.0, -1.0)
    end = torch.trunc(u + du + us)
    live = torch.nonzero(out > 0).reshape(-1)
    u, v, du, dv, us, vs, end, steep = (a[live] for a in (u, v, du, dv, us, vs, end, steep))
    u0, v0, err, du, dv = u, v, torch.zeros_like(u), du.abs(), dv.abs()
    while len(live):
        u = u + us
        err = err + dv
        up = err * 2.0 >= du
        v, err = torch.where(up, v + vs, v), torch.where(up, err - du, err)
        hit = occupied(torch.where(steep, u, v), torch.where(steep, v, u))
        out[live[hit]] = torch.sqrt((u - u0) ** 2 + (v - v0) ** 2)[hit]
        go = ~hit & (torch.trunc(u) != end)
        live, u, v, du, dv, us, vs, end, steep, u0, v0, err = (
            a[go] for a in (live, u, v, du, dv, us, vs, end, steep, u0, v0, err))
    return out


def _cddt64(occ, x, y, th, mr, td):
    """The compressed directional table of `occ` and its queries: zero points as (bin, position)
    pairs of one sorted list."""
    o = torch.from_numpy(occ != 0).to(DEV)
    W_, H_ = o.shape
    pad = torch.nn.functional.pad(o[None, None].float(), (1, 1, 1, 1), value=1.0)
    near_free = -torch.nn.functional.max_pool2d(-pad, 3, 1)[0, 0] < 0.5
    ex, ey = [a.double() + 0.5 for a in torch.nonzero(o & near_free, as_tuple=True)]
    angle = torch.arange(td, device=DEV).double() * (M_2PI / td)
    ca, sa = torch.cos(angle), torch.sin(angle)
    width = torch.ceil(W_ * sa.abs() + H_ * ca.abs() - 1e-5).long()
    low = torch.minimum(torch.minimum(W_ * sa, W_ * sa + H_ * ca), H_ * ca)
    trans = torch.clamp(-low - 1e-5, min=0.0)
    base = torch.cumsum(width, 0) - width
    span = 16384.0                                   # more than any position's range
    keys = []
    for a in range((td + 1) // 2):
        half = (sa[a].abs() + ca[a].abs()) / 2
        lx, ly = ex * ca[a] - ey * sa[a], ex * sa[a] + ey * ca[a] + trans[a]
        lo, hi = torch.trunc(ly - half + 1e-5).long(), torch.trunc(ly + half - 1e-5).long()
        for k in range(3):
            b = lo + k
            ok = (b <= hi) & (b >= 0) & (b < width[a])
            keys.append(((b + base[a]).double() * span + lx)[ok])
    zeros = torch.sort(torch.cat(keys)).values
    th = torch.remainder(-th, M_2PI)
    flip = th >= math.pi
    a = torch.round(torch.where(flip, th - math.pi, th) * td / M_2PI).long()
    half_turn = a == td // 2
    a, flip = torch.where(half_turn, 0, a) % td, flip ^ half_turn
    lx, ly = x * ca[a] - y * sa[a], x * sa[a] + y * ca[a] + trans[a]
    li = torch.trunc(ly).long()
    inside = (li >= 0) & (li < width[a])
    here = (torch.where(inside, li, 0) + base[a]).double() * span
    at = torch.searchsorted(zeros, here + lx)
    last = len(zeros) - 1
    after, before = zeros[at.clamp(max=last)], zeros[(at - 1).clamp(min=0)]
    has_after = (at <= last) & (after < here + span / 2)
    has_before = (at > 0) & (before > here - span / 2)
    px, py = torch.trunc(x).long(), torch.trunc(y).long()
    on_map = (px >= 0) & (px < W_) & (py >= 0) & (py < H_)
    filled = on_map & o.reshape(-1)[torch.where(on_map, px * H_ + py, 0)]
    r = torch.where(flip, torch.where(has_before, here + lx - before, mr), torch.where(has_after, after - here - lx, mr))
    r = torch.where(filled & has_before & has_after, 0.0, r)   # inside a wall, between two of its edges
    return torch.where(inside, r, mr)


def _glt64(dt, x, y, th, mr, td):
    W_, H_ = dt.shape
    b = torch.round(torch.remainder(th, M_2PI) * td / M_2PI).long() % td
    ang = b.double() * (M_2PI / td)
    px, py = torch.trunc(x), torch.trunc(y)
    r = _march64(dt, px, py, torch.cos(ang), torch.sin(ang), mr).clamp(max=mr)
    r = torch.trunc(r * 65535.0 / mr) * mr / 65535.0
    return torch.where((x >= 0) & (x < W_) & (y >= 0) & (y < H_), r, mr)


def _ranges64(kind, d, mr, td):
    """Pixel ranges of the inputs' rays."""
    x, y, th = _grid_rays(d["ins"], d.get("angles"), d["world"])
    if kind == "cddt":
        return _cddt64(d["occ"], x, y, th, mr, td)
    if kind == "bl":
        return _walk64(d["occ"], x, y, torch.cos(th), torch.sin(th), mr)
    dt = _edt64(d["occ"])
    if kind == "glt":
        return _glt64(dt, x, y, th, mr, td)
    return _march64(dt, x, y, torch.cos(th), torch.sin(th), mr)


def _weights64(d, ranges):
    """Products over each particle's beams of table[observed bin, expected bin]."""
    table = torch.from_numpy(d["table"]).to(DEV)
    K = len(table)
    # the library multiplies by the float nearest to 1 / scale and bins what that gives
    obs = (torch.from_numpy(d["obs"]).to(DEV) * float(np.float32(1.0 / np.float32(d["world"][0])))).double()
    row = obs.clamp(0, K - 1).long()
    col = ranges.clamp(0, K - 1).long().reshape(-1, len(row))
    w = torch.ones(len(col), dtype=torch.float64, device=DEV)
    for a in range(len(row)):
        w = w * table[row[a], col[:, a]]
    return w


def exact(case, seed):
    f = case["family"]
    kind = case.get("kind", "rm")
    if f == "learned_train":      # Adam steps of a 16-bit network: its rounding is the computation
        return None
    if f == "batch":
        got = []
        for spec in _specs(case):
            d = _filter_inputs(spec, seed)
            got.append(_weights64(d, _ranges64("rm", d, spec.max_range, 0)))
        return got
    if kind == "pcddt" or f == "learned_query":
        # which zero points a pruned table keeps, and which predictions pass the check, hang on the
        # last bit of what was computed in 32 and 16 bits; both are compared with the start alone
        return None
    d = _inputs(case, seed)
    r = _ranges64(kind, d, case["max_range"], case.get("td") or 108)
    if f == "pf":
        return _weights64(d, r)
    scale = d["world"][0]
    if f == "plain":
        # a range that lies on a bin's edge may fall to either side of it: the weights are those of
        # the ranges as they are handed over, in 32 bits
        handed = (r * scale).float() * float(np.float32(1.0 / np.float32(scale)))
        return {"ranges": r * scale, "weights": _weights64(d, handed.double())}
    return r * scale

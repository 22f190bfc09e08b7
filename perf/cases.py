"""The work that programs have this engine do, as cases to measure.

A pass is one frame of a program that owns the state on the host: the state of
every world goes up from pinned memory, ``update`` advances it by one frame,
and the new state comes down to pinned memory.  All of it is queued on one
stream; nothing waits.  A program with one world calls ``Solver.update``, one
with many independent worlds ``Batch.update``.

A case says what the worlds hold (``kind``), how much of it, and the solver's
options: sub-steps, link iterations, link order (reference or fast), stiffness
and collisions.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bendy2d_gb300 import api

F32 = np.float32
DT = 1.0 / 60.0
GRAVITY = (0.0, -9.81)
ALL = api.COLLIDE_PP | api.COLLIDE_PC | api.COLLIDE_PPOLY


# ---------------------------------------------------------------- the cases
def listed() -> list:
    return [
        # a small soft body with the reference's own settings (one sub-step,
        # one link pass): the smallest call a game makes every frame
        {"name": "cloth_8x8_defaults", "kind": "cloth", "bodies": 1, "w": 8, "h": 8, "sub": 1,
         "iters": 1, "fast": False, "stiff": False},
        # one cloth with circles and a floor, reference link order: the
        # ordinary soft body
        {"name": "cloth_32x32", "kind": "cloth", "bodies": 1, "w": 32, "h": 32, "sub": 8,
         "iters": 4, "fast": False, "stiff": False},
        # a few odd-sized cloths with stiffness, fast link order
        {"name": "cloth_3x41x27_fast", "kind": "cloth", "bodies": 3, "w": 41, "h": 27, "sub": 8,
         "iters": 4, "fast": True, "stiff": True},
        # one body larger than a CTA's shared memory
        {"name": "cloth_100x100", "kind": "cloth", "bodies": 1, "w": 100, "h": 100, "sub": 8,
         "iters": 4, "fast": False, "stiff": False},
        # ropes and bridges: chain-like bodies
        {"name": "ropes_24x200", "kind": "ropes", "ropes": 24, "length": 200, "sub": 8,
         "iters": 4},
        # circles and polygons only: the reference's dynamic bodies
        {"name": "rigid_48c_24p", "kind": "rigid", "circles": 48, "polygons": 24, "sub": 8},
        # link-free particles that collide (granular matter)
        {"name": "grains_50021", "kind": "grains", "n": 50021, "sub": 4},
        # the benchmark scene: 64 cloths, particle collisions, circles, polygons
        {"name": "scene_64_cloths", "kind": "scene", "bodies": 64, "w": 32, "h": 32, "sub": 8,
         "iters": 4, "fast": False, "packed": False, "circles": 16, "polygons": 8},
        # the stress scene's settings (lattice, fast link order, 20 sub-steps, 8
        # link passes) with more bodies than the GPU has multiprocessors
        {"name": "scene_200_cloths_fast", "kind": "scene", "bodies": 200, "w": 32, "h": 32,
         "sub": 20, "iters": 8, "fast": True, "packed": True, "circles": 24, "polygons": 12},
        # many independent worlds of hub-and-spoke rings in one batch
        {"name": "batch_400_rings", "kind": "rings", "worlds": 400, "lo": 64, "hi": 4096,
         "iters": 1},
        # one serving tick: collision worlds of very different sizes
        {"name": "batch_40_requests", "kind": "requests", "worlds": 40, "lo": 64, "hi": 16384},
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["cloth", "cloth", "scene", "scene", "ropes", "rigid", "grains", "rings",
                       "requests"])
    if kind == "cloth":  # up to ~16 k particles over the bodies
        w, h = _log_int(rng, 3, 110), _log_int(rng, 3, 110)
        return {"kind": kind, "bodies": _log_int(rng, 1, max(1, min(24, 16000 // (w * h)))),
                "w": w, "h": h, "sub": rng.choice([1, 2, 3, 4, 8]),
                "iters": rng.choice([1, 2, 4]), "fast": rng.random() < 0.4,
                "stiff": rng.random() < 0.4}
    if kind == "ropes":
        return {"kind": kind, "ropes": _log_int(rng, 1, 300), "length": _log_int(rng, 4, 700),
                "sub": rng.choice([1, 3, 4, 8]), "iters": rng.choice([1, 2, 4])}
    if kind == "rigid":
        return {"kind": kind, "circles": _log_int(rng, 2, 40), "polygons": _log_int(rng, 1, 40),
                "sub": rng.choice([1, 2, 5, 8])}
    if kind == "grains":
        return {"kind": kind, "n": _log_int(rng, 50, 200000), "sub": rng.choice([1, 2, 4, 7])}
    if kind == "scene":
        w, h = _log_int(rng, 8, 48), _log_int(rng, 8, 48)
        return {"kind": kind, "bodies": _log_int(rng, 2, max(2, min(240, 200000 // (w * h)))),
                "w": w, "h": h, "sub": rng.choice([2, 5, 8]), "iters": rng.choice([1, 4, 6]),
                "fast": rng.random() < 0.5, "packed": rng.random() < 0.5,
                "circles": rng.randint(0, 40), "polygons": rng.randint(0, 24)}
    if kind == "rings":
        return {"kind": kind, "worlds": _log_int(rng, 1, 400), "lo": 64,
                "hi": _log_int(rng, 200, 4096), "iters": rng.choice([1, 2])}
    return {"kind": kind, "worlds": _log_int(rng, 2, 60), "lo": 64,
            "hi": _log_int(rng, 500, 16384)}


# --------------------------------------------------------------- the worlds
def _grid(w, h, n=None):
    """Points and links of a w x h cloth: structural links row by row (right,
    then down), then both diagonals of each cell; its first n points only."""
    y, x = (a.ravel() for a in np.mgrid[0:h, 0:w])
    i = y * w + x
    a = np.stack([i, i], 1)
    b = np.stack([i + 1, i + w], 1)
    ok = np.stack([x + 1 < w, y + 1 < h], 1)
    cy, cx = (v.ravel() for v in np.mgrid[0:h - 1, 0:w - 1])
    c = cy * w + cx
    la = np.concatenate([a[ok], np.stack([c, c + 1], 1).ravel()])
    lb = np.concatenate([b[ok], np.stack([c + w + 1, c + w], 1).ravel()])
    pos = np.stack([x, y], 1).astype(np.float64)
    if n is not None:
        keep = (la < n) & (lb < n)
        pos, la, lb = pos[:n], la[keep], lb[keep]
    return pos, la, lb


def _ring(n, radius):
    """n rim points and a hub: rim links, then spokes."""
    th = 2.0 * np.pi * np.arange(n) / n
    pos = np.vstack([radius * np.stack([np.cos(th), np.sin(th)], 1), np.zeros((1, 2))])
    i = np.arange(n)
    j = (i + 1) % n
    return pos, np.concatenate([np.minimum(i, j), i]), np.concatenate([np.maximum(i, j),
                                                                       np.full(n, n)])


def _world(rng, bodies, *, box, sub, iters, fast=False, collide=0, circles=(), polygons=(),
           speed=0.0, stiff=None):
    """A world of link-connected bodies [(points, a, b)]: rest lengths are the
    initial distances, velocities are normal with deviation `speed`."""
    at = np.cumsum([0] + [len(p) for p, _, _ in bodies])
    none = np.zeros(0, np.int64)
    pos = np.vstack([p for p, _, _ in bodies] or [np.zeros((0, 2))]).astype(F32)
    la = np.concatenate([a + o for (_, a, _), o in zip(bodies, at)] or [none])
    lb = np.concatenate([b + o for (_, _, b), o in zip(bodies, at)] or [none])
    d = pos[la] - pos[lb]
    prev = pos - rng.normal(0.0, speed, pos.shape) * (DT / sub) if speed else pos
    return {"pos": pos, "prev": prev.astype(F32), "la": la, "lb": lb,
            "rest": np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]),
            "stiff": None if stiff is None else np.asarray(stiff, F32), "box": float(box),
            "sub": sub, "iters": iters, "fast": fast, "collide": collide,
            "circles": list(circles), "polygons": list(polygons)}


def _circles(rng, n, box, lo, hi, static):
    return [(rng.uniform(0.0, box, 2).astype(F32), float(F32(rng.uniform(lo, hi))), static)
            for _ in range(n)]


def _polygon(rng, n, center, radius):
    th = np.sort(rng.uniform(0.0, 2.0 * np.pi, n))
    return (np.asarray(center) + radius * np.stack([np.cos(th), np.sin(th)], 1)).astype(F32)


def _floor(box, depth):
    return (np.array([[0, 0], [box, 0], [box, depth], [0, depth]], F32), True)


def _jittered(rng, body, origin):
    pos, a, b = body
    return pos + np.asarray(origin) + rng.uniform(-0.01, 0.01, pos.shape), a, b


def _worlds(case, seed) -> list:
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "cloth":
        w, h, n = case["w"], case["h"], case["bodies"]
        box = 100.0 + 1.5 * max(w, h) * math.ceil(math.sqrt(n))
        body = _grid(w, h)
        bodies = [_jittered(rng, body, rng.uniform(5.0, box - 5.0 - max(w, h), 2))
                  for _ in range(n)]
        stiff = rng.uniform(0.3, 1.0, n).repeat(len(body[1])) if case["stiff"] else None
        return [_world(rng, bodies, box=box, sub=case["sub"], iters=case["iters"],
                       fast=case["fast"], stiff=stiff, speed=0.5,
                       circles=_circles(rng, 4, box, 5.0, 5.0, True), polygons=[_floor(box, 4)])]
    if kind == "ropes":
        k = case["length"]
        i = np.arange(k - 1)
        body = (np.stack([np.arange(k), np.zeros(k)], 1), i, i + 1)
        box = 100.0 + 1.2 * k
        bodies = [_jittered(rng, body, (rng.uniform(5.0, box - 5.0 - k), rng.uniform(20, box - 5)))
                  for _ in range(case["ropes"])]
        return [_world(rng, bodies, box=box, sub=case["sub"], iters=case["iters"], speed=0.5,
                       polygons=[_floor(box, 4)])]
    if kind == "rigid":
        nc, ng = case["circles"], case["polygons"]
        box = 20.0 * math.sqrt(nc + 2 * ng) + 40.0
        polys = [(_polygon(rng, 4 + k % 5, rng.uniform(12.0, box - 12.0, 2),
                           rng.uniform(4.0, 10.0)), False) for k in range(ng)]
        return [_world(rng, [], box=box, sub=case["sub"], iters=1,
                       circles=_circles(rng, nc, box, 2.0, 8.0, False), polygons=polys)]
    if kind == "grains":
        n = case["n"]
        box = math.ceil(math.sqrt(2.0 * n)) + 4.0
        none = np.zeros(0, np.int64)
        return [_world(rng, [(rng.uniform(0.0, box, (n, 2)), none, none)], box=box,
                       sub=case["sub"], iters=1, collide=api.COLLIDE_PP, speed=0.5)]
    if kind == "scene":
        n, size = case["bodies"], max(case["w"], case["h"])
        pitch = size * (3.8 if case["packed"] else 7.8)
        side = math.ceil(math.sqrt(n))
        box = 100.0 + pitch * side
        body = _grid(case["w"], case["h"])
        at = ([(50.0 + pitch * (k % side), 50.0 + pitch * (k // side)) for k in range(n)]
              if case["packed"] else rng.uniform(0.0, box - size, (n, 2)))
        polys = [(_polygon(rng, 4 + k % 5, rng.uniform(50.0, box - 50.0, 2),
                           rng.uniform(10.0, 50.0)), case["packed"])
                 for k in range(case["polygons"])]
        return [_world(rng, [_jittered(rng, body, o) for o in at], box=box, sub=case["sub"],
                       iters=case["iters"], fast=case["fast"], collide=ALL, speed=0.5,
                       circles=_circles(rng, case["circles"], box, 5.0, 30.0, case["packed"]),
                       polygons=polys)]
    # particle counts spread evenly over their logarithm, in a fixed shuffled order
    k = case["worlds"]
    sizes = np.exp(np.linspace(np.log(case["lo"]), np.log(case["hi"]), k + 2)[1:-1]).astype(int)
    sizes = sizes[np.random.default_rng(k).permutation(k)]
    if kind == "rings":  # 1-8 rings of equal size a world
        out = []
        for i, n in enumerate(sizes):
            k = 1 + i % 8
            bodies, stiff = [], []
            for _ in range(k):
                r = rng.uniform(5.0, 20.0)
                p, a, b = _ring(int(n) // k - 1, r)
                bodies.append((p + rng.uniform(r + 5.0, 995.0 - r, 2), a, b))
                stiff.append(np.full(len(a), rng.uniform(0.3, 1.0)))
            out.append(_world(rng, bodies, box=1000.0, sub=8, iters=case["iters"],
                              stiff=np.concatenate(stiff), polygons=[_floor(1000, 10)],
                              circles=_circles(rng, 2, 1000.0, 5.0, 20.0, False)))
        return out
    out = []  # requests: 32-wide cloths, the last one partial
    for n in sizes:
        bodies, left = [], int(n)
        while left > 0:
            k = min(left, 1024)
            bodies.append(_jittered(rng, _grid(32, (k + 31) // 32, k),
                                    rng.uniform(0.0, 1968.0, 2)))
            left -= k
        out.append(_world(rng, bodies, box=2000.0, sub=8, iters=4, collide=api.COLLIDE_PP,
                          speed=0.5))
    return out


# ------------------------------------------------------------- the programs
_stream = None


def _the_stream():
    """The one stream on which the program queues its simulation."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def _solver(w) -> api.Solver:
    s = api.Solver()
    s.gravity = GRAVITY
    s.bounds = api.Bounds((0.0, 0.0), (w["box"], w["box"]))
    s.set_sub_steps(w["sub"])
    s.set_link_iters(w["iters"])
    s.set_mode(api.MODE_FAST if w["fast"] else api.MODE_REFERENCE)
    s.set_collision(w["collide"], 0.5, 1.0)
    s.add_particles(w["pos"], w["prev"])
    if len(w["la"]):
        s.add_particle_links(w["la"], w["lb"], w["rest"], w["stiff"])
    for p, radius, static in w["circles"]:
        s.add_circle(api.Circle(api.Particle.new(p), radius, static))
    for pts, static in w["polygons"]:
        s.add_polygon_points(pts, static)
    return s


def prepare(case, seed):
    solvers = [_solver(w) for w in _worlds(case, seed)]
    many = api.Batch(solvers) if case["kind"] in ("rings", "requests") else None
    (many or solvers[0]).set_stream(_the_stream())
    sizes = [s.state_bytes() // 4 for s in solvers]
    at = np.cumsum([0] + sizes)
    src = torch.empty(int(at[-1]), dtype=torch.float32, pin_memory=True)
    out = torch.empty_like(src, pin_memory=True)
    for s, o in zip(solvers, at):
        s.state_download_async(src.data_ptr() + 4 * int(o))
    torch.cuda.synchronize()
    return {"solvers": solvers, "update": (many or solvers[0]).update, "many": many, "src": src,
            "out": out, "up": [src.data_ptr() + 4 * int(o) for o in at[:-1]],
            "down": [out.data_ptr() + 4 * int(o) for o in at[:-1]]}


def run(state):
    for s, p in zip(state["solvers"], state["up"]):
        s.state_upload_async(p)
    state["update"](DT)
    for s, p in zip(state["solvers"], state["down"]):
        s.state_download_async(p)
    return {"state": state["out"]}


def work(case):
    """The state read and written once, each link's endpoints, rest length and
    stiffness read once; ~30 flops per link solve, ~14 per bounds + integrate."""
    size = flops = 0
    for w in _worlds(case, 0):
        rigid = 3 * len(w["circles"]) + sum(3 * len(p) + 1 for p, _ in w["polygons"])
        size += 2 * 8 * (2 * len(w["pos"]) + rigid) + 16 * len(w["la"])
        flops += w["sub"] * (30 * w["iters"] * len(w["la"]) + 14 * (len(w["pos"]) + rigid))
    return {"bytes": size, "flops": flops}


# ------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """What run() returns, computed in 64 bits with numpy: the links of all
    worlds level by level (a level's links share no particle, and each particle
    meets its links in order), contacts on a sorted grid, circles and polygons
    one pair after another."""
    ws = _worlds(case, seed)
    S, iters = ws[0]["sub"], ws[0]["iters"]
    n = [len(w["pos"]) for w in ws]
    links = sum(len(w["la"]) for w in ws)
    if S * (iters * links + 8 * sum(n) * bool(ws[0]["collide"])) > 30e6:
        return None  # minutes of numpy
    at = np.cumsum([0] + n)
    p = np.vstack([w["pos"] for w in ws]).astype(np.float64)
    q = np.vstack([w["prev"] for w in ws]).astype(np.float64)
    a = np.concatenate([w["la"] + o for w, o in zip(ws, at)])
    b = np.concatenate([w["lb"] + o for w, o in zip(ws, at)])
    rest = np.concatenate([w["rest"] for w in ws]).astype(np.float64)
    stiff = np.concatenate([np.ones(len(w["la"])) if w["stiff"] is None else w["stiff"]
                            for w in ws]).astype(np.float64)
    if ws[0]["fast"]:
        order = np.argsort(_colours(a, b, len(p)), kind="stable")
        a, b, rest, stiff = a[order], b[order], rest[order], stiff[order]
    level = _levels(a, b, len(p))
    order = np.argsort(level, kind="stable")
    ends = np.cumsum(np.bincount(level)) if len(level) else []
    a, b, rest, stiff = a[order], b[order], rest[order], stiff[order]
    which = np.repeat(np.arange(len(ws)), n)
    rigid = [_Rigid(w) for w in ws]
    h = float(F32(DT) * (F32(1.0) / F32(S)))
    g = np.asarray(GRAVITY, F32).astype(np.float64)
    box = ws[0]["box"]
    for _ in range(S):
        for r in rigid:
            r.forces_and_contacts(g, iters)
        for _ in range(iters):
            lo = 0
            for hi in ends:
                i, j = a[lo:hi], b[lo:hi]
                pi, pj = p[i], p[j]
                d = pi - pj
                dist = np.sqrt((d * d).sum(1))
                c = d * ((dist - rest[lo:hi]) / dist * 0.5 * stiff[lo:hi])[:, None]
                p[i] = pi - c
                p[j] = pj + c
                lo = hi
        collide = ws[0]["collide"]
        if collide & api.COLLIDE_PP:
            p = _contacts(p, which, 1.0, 1.0)
        if collide & (api.COLLIDE_PC | api.COLLIDE_PPOLY):
            p = rigid[0].push(p, 0.5)
        p, q = _bounds(p, q, 0.0, box)
        p, q = p + (p - q) + g * h * h, p
        for r in rigid:
            r.bounds_and_move(box, h)
    parts = []
    for k, r in enumerate(rigid):
        s = slice(at[k], at[k + 1])
        parts += [p[s].ravel(), q[s].ravel(), r.flat()]
    return {"state": np.concatenate(parts)}


def _levels(a, b, n):
    last, out = [0] * n, np.empty(len(a), np.int64)
    for k, (i, j) in enumerate(zip(a.tolist(), b.tolist())):
        v = max(last[i], last[j])
        out[k] = v
        last[i] = last[j] = v + 1
    return out


def _colours(a, b, n):
    """Each link takes the first colour that neither of its ends has yet."""
    used, out = [0] * n, np.empty(len(a), np.int64)
    for k, (i, j) in enumerate(zip(a.tolist(), b.tolist())):
        free = ~(used[i] | used[j])
        bit = free & -free
        out[k] = bit.bit_length() - 1
        used[i] |= bit
        used[j] |= bit
    return out


def _bounds(p, q, lo, hi):
    lo, hi = np.broadcast_to(lo, p.shape), np.broadcast_to(hi, p.shape)
    edge = np.where(p < lo, lo, np.where(p > hi, hi, p))
    return edge, np.where(edge != p, edge - (q - p), q)


def _contacts(p, which, cell, diameter):
    """Every overlapping pair of one world pushed apart by half the overlap
    each, all from the same positions."""
    c = np.floor(p / cell).astype(np.int64)
    key = (which * (1 << 40)) + ((c[:, 1] + (1 << 18)) << 20) + (c[:, 0] + (1 << 18))
    order = np.argsort(key, kind="stable")
    key = key[order]
    move = np.zeros_like(p)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            want = key + (dy << 20) + dx
            lo = np.searchsorted(key, want, "left")
            hi = np.searchsorted(key, want, "right")
            k = 0
            while True:
                i = np.nonzero(lo + k < hi)[0]
                if not len(i):
                    break
                me, other = order[i], order[lo[i] + k]
                d = p[me] - p[other]
                d2 = (d * d).sum(1)
                hit = (d2 < diameter * diameter) & (d2 > 0.0)
                dist = np.sqrt(d2[hit])
                # one other a round, so `me` holds no particle twice
                move[me[hit]] += d[hit] * ((diameter - dist) / dist * 0.5)[:, None]
                k += 1
    return p + move


def _cross(p1, p2, p3, p4):
    """Where the segments p1-p2 and p3-p4 meet, or None."""
    ax, ay = p2[0] - p1[0], p2[1] - p1[1]
    bx, by = p4[0] - p3[0], p4[1] - p3[1]
    dx, dy = p1[0] - p3[0], p1[1] - p3[1]
    den = ax * by - bx * ay
    if den == 0.0:
        return None
    s, t = (ax * dy - ay * dx) / den, (bx * dy - by * dx) / den
    if 0.0 <= s <= 1.0 and 0.0 <= t <= 1.0:
        return p1[0] + t * ax, p1[1] + t * ay
    return None


def _edge_hit(center, a, b, v, other):
    """Vertex v of a polygon with centre `other` against the edge a-b of one
    with centre `center`: the new a, b and v, or None."""
    hit = _cross(a, b, v, other)
    if hit is None:
        return None
    ex, ey = b[0] - a[0], b[1] - a[1]
    along = ((center[0] - hit[0]) * ex + (center[1] - hit[1]) * ey) / (ex * ex + ey * ey)
    nx, ny = center[0] - hit[0] - along * ex, center[1] - hit[1] - along * ey
    size = math.hypot(nx, ny)
    if size == 0.0:
        return None
    nx, ny = nx / size, ny / size
    da, db = math.dist(hit, a), math.dist(hit, b)
    depth = (nx * (hit[0] - v[0]) + ny * (hit[1] - v[1])) * 2.0 / 3.0
    wa, wb = depth * db / (da + db), depth * da / (da + db)
    out = _cross(a, b, v, (v[0] - nx * 1e4, v[1] - ny * 1e4))
    if out is None:
        return None
    return (a[0] - nx * wa, a[1] - ny * wa), (b[0] - nx * wb, b[1] - ny * wb), out


class _Rigid:
    """The circles and polygons of one world."""

    def __init__(self, w):
        self.cp = np.array([c[0] for c in w["circles"]], np.float64).reshape(-1, 2)
        self.cq, self.ca = self.cp.copy(), np.zeros_like(self.cp)
        self.r = np.array([c[1] for c in w["circles"]], np.float64)
        self.fixed = np.array([c[2] for c in w["circles"]], bool)
        self.v = [pts.astype(np.float64) for pts, _ in w["polygons"]]
        self.vq = [v.copy() for v in self.v]
        self.va = [np.zeros_like(v) for v in self.v]
        self.still = [static for _, static in w["polygons"]]
        self.center = [v.mean(0) for v in self.v]
        self.links = []
        for v in self.v:
            e = [(min(i, (i + 1) % len(v)), max(i, (i + 1) % len(v))) for i in range(len(v))]
            self.links.append([(i, j, math.dist(v[i], v[j])) for i, j in e])

    def forces_and_contacts(self, g, iters):
        self.ca += g
        for acc in self.va:
            acc += g
        for _ in range(iters):
            for k, v in enumerate(self.v):
                self.center[k] = v.mean(0)
                for i, j, rest in self.links[k]:
                    d = v[i] - v[j]
                    dist = math.hypot(d[0], d[1])
                    c = d * ((dist - rest) / dist * 0.5)
                    v[i] -= c
                    v[j] += c
        cp, r = self.cp, self.r
        for i in range(len(cp) - 1):
            for j in range(i + 1, len(cp)):
                dx, dy = cp[i, 0] - cp[j, 0], cp[i, 1] - cp[j, 1]
                d2, both = dx * dx + dy * dy, r[i] + r[j]
                if d2 < both * both:
                    dist = math.sqrt(d2)
                    f = (both - dist) / dist / (r[i] * r[i] + r[j] * r[j])
                    move = np.array([dx * f, dy * f])
                    cp[i] += move * (r[j] * r[j])
                    cp[j] -= move * (r[i] * r[i])
        v = [[tuple(x) for x in v.tolist()] for v in self.v]
        c = [tuple(x) for x in self.center]
        for i in range(len(v)):
            for j in range(i + 1, len(v)):
                for one, two in ((i, j), (j, i)):
                    for e in range(len(v[one])):
                        f = (e + 1) % len(v[one])
                        a, b = v[one][e], v[one][f]
                        for k in range(len(v[two])):
                            hit = _edge_hit(c[one], a, b, v[two][k], c[two])
                            if hit is not None:
                                v[one][e], v[one][f], v[two][k] = hit
        self.v = [np.array(x).reshape(-1, 2) for x in v]

    def push(self, p, radius):
        """Particles of the given radius pushed out of circles, then polygons."""
        for c, r in zip(self.cp, self.r):
            d = p - c
            d2 = (d * d).sum(1)
            i = np.nonzero((d2 < (r + radius) ** 2) & (d2 > 0.0))[0]
            dist = np.sqrt(d2[i])
            p[i] += d[i] * ((r + radius - dist) / dist)[:, None]
        for v in self.v:
            near = ((p >= v.min(0) - radius) & (p <= v.max(0) + radius)).all(1)
            i = np.nonzero(near)[0]
            x = p[i]
            inside = np.zeros(len(i), bool)
            best, foot = np.full(len(i), np.inf), x.copy()
            for e in range(len(v)):
                a, b = v[e], v[(e + 1) % len(v)]
                ab = b - a
                spans = (a[1] > x[:, 1]) != (b[1] > x[:, 1])
                with np.errstate(divide="ignore", invalid="ignore"):
                    cut = a[0] + (x[:, 1] - a[1]) / ab[1] * ab[0]
                inside ^= spans & (x[:, 0] < cut)
                f = a + ab * np.clip((x - a) @ ab / (ab @ ab), 0.0, 1.0)[:, None]
                d2 = ((x - f) ** 2).sum(1)
                less = d2 < best
                best, foot[less] = np.where(less, d2, best), f[less]
            k = np.nonzero((inside | (best < radius * radius)) & (best > 0.0))[0]
            out = np.where(inside[k, None], foot[k] - x[k], x[k] - foot[k])
            p[i[k]] = foot[k] + out * (radius / np.sqrt(best[k]))[:, None]
        return p

    def bounds_and_move(self, box, h):
        r = self.r[:, None]
        self.cp, self.cq = _bounds(self.cp, self.cq, r, box - r)
        go = ~self.fixed
        p = self.cp.copy()
        self.cp[go] += p[go] - self.cq[go] + self.ca[go] * h * h
        self.cq[go], self.ca[go] = p[go], 0.0
        for k, v in enumerate(self.v):
            v, q = _bounds(v, self.vq[k], 0.0, box)
            if not self.still[k]:
                self.center[k] = v.mean(0)
                v, q = v + (v - q) + self.va[k] * h * h, v
                self.va[k] = np.zeros_like(v)
            self.v[k], self.vq[k] = v, q

    def flat(self):
        parts = [self.cp, self.cq, self.ca] + self.v + self.vq + self.va + self.center
        return np.concatenate([np.asarray(x).ravel() for x in parts] or [np.zeros(0)])

"""Performance cases of the simulation framework, one per way a program uses it.

A case is a dict of plain values.  `prepare` builds what a user's program holds before
the call (the world or server, page-locked body arrays, query records), `run` is one call
sequence through the public API and returns everything it produced, `work` states the
least memory traffic and arithmetic of that call, and `exact` evaluates ray queries in
64-bit arithmetic.

A frame changes the state it starts from, so `run` starts every pass from the same state:
the bodies' state lives in host arrays (the caller's registry), as
`World.simulate_host` and `World.write_bodies` expect it.
"""
import copy
import math

import numpy as np
import torch

from physecs_gb300 import scenes as gen
from physecs_gb300.api import Server, World, trimesh_build
from physecs_gb300.desc import make_desc

KEYS = ("pos", "quat", "vel", "ang_vel")
HULLS = 8                     # convex hulls shared by the bodies of a batched scene
TEMPLATES = 256               # distinct scenes of a batch; the rest are copies with velocities of their own
# slots of the serving cases: (bodies, slots), for requests of up to 1000 bodies
SERVE_CLASSES = [(17, 48), (33, 48), (65, 48), (129, 48), (257, 32), (513, 24), (1025, 16)]


def listed():
    return [
        # an interactive application's smallest scene: a handful of bodies, one frame at a
        # time between its own reads and writes; launches and latency are all there is
        {"name": "frame_mixed_16", "kind": "frame", "scene": "mixed", "bodies": 16},
        # the 20-row box pyramid: one stacked scene, a long chain of dependent contacts
        {"name": "frame_pyramid_20", "kind": "frame", "scene": "pyramid", "rows": 20},
        # one ordinary scene of mixed shapes, larger than a single block's share
        {"name": "frame_mixed_2000", "kind": "frame", "scene": "mixed", "bodies": 2000},
        # a large open world: 65,536 bodies landing on a terrain of 131,072 triangles
        {"name": "frame_terrain_65536", "kind": "frame", "scene": "terrain", "bodies": 65536, "cells": 256},
        # articulated bodies: 2048 swinging chains of 32 links with every joint kind of the demo
        {"name": "frame_chains_2048x32", "kind": "frame", "scene": "chains", "chains": 2048, "links": 32},
        # sample collection: independent scenes stepped several frames between two reads
        {"name": "rollout_256x8", "kind": "rollout", "scenes": 256, "frames": 8},
        # the throughput workload: 4096 independent scenes, one frame end to end
        {"name": "batch_4096", "kind": "batch", "scenes": 4096},
        # continuous batching: requests of 8 to 1000 bodies arrive, run and leave
        {"name": "serve_48", "kind": "serve", "requests": 48, "per_tick": 3, "max_bodies": 1000, "max_frames": 24},
        # range sensors: many rays against many scenes
        {"name": "rays_65536", "kind": "rays", "rays": 65536, "scenes": 64, "bodies": 200},
        # a game server's frame: every scene's character moves, then the scenes step
        {"name": "characters_128", "kind": "characters", "scenes": 128, "balls": 100},
        # loading a terrain tile: the triangle mesh and its tree from vertices and indices
        {"name": "terrain_build_256", "kind": "trimesh", "cells": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "pyramid", "terrain", "chains", "rollout", "batch", "batch", "serve", "rays",
                       "characters", "trimesh"])
    if kind == "mixed":
        return {"kind": "frame", "scene": "mixed", "bodies": _log_int(rng, 8, 4096)}
    if kind == "pyramid":
        return {"kind": "frame", "scene": "pyramid", "rows": _log_int(rng, 2, 30)}
    if kind == "terrain":
        return {"kind": "frame", "scene": "terrain", "bodies": _log_int(rng, 1024, 65536), "cells": _log_int(rng, 96, 256)}
    if kind == "chains":
        return {"kind": "frame", "scene": "chains", "chains": _log_int(rng, 8, 2048), "links": _log_int(rng, 2, 32)}
    if kind == "rollout":
        return {"kind": "rollout", "scenes": _log_int(rng, 8, 512), "frames": rng.randint(2, 8)}
    if kind == "batch":
        return {"kind": "batch", "scenes": _log_int(rng, 16, 4096)}
    if kind == "serve":
        return {"kind": "serve", "requests": _log_int(rng, 4, 48), "per_tick": rng.randint(1, 4),
                "max_bodies": _log_int(rng, 100, 1000), "max_frames": rng.randint(4, 24)}
    if kind == "rays":
        return {"kind": "rays", "rays": _log_int(rng, 64, 65536), "scenes": _log_int(rng, 1, 64),
                "bodies": _log_int(rng, 16, 400)}
    if kind == "characters":
        return {"kind": "characters", "scenes": _log_int(rng, 1, 128), "balls": _log_int(rng, 8, 150)}
    return {"kind": "trimesh", "cells": _log_int(rng, 4, 384)}


# ---------------------------------------------------------------- scenes

def _pool():
    return gen._hull_pool(gen.SplitMix64(gen.scene_seed(4, 1 << 19)), count=HULLS)


def _with_velocity(s, rng, sigma):
    """A copy of scene `s` whose dynamic bodies get random velocities."""
    c = copy.copy(s)
    c.arrays = dict(s.arrays)
    moving = (s.arrays["flags"] & gen.BODY_DYNAMIC) != 0
    for k in ("vel", "ang_vel"):
        c.arrays[k] = (s.arrays[k] + sigma * rng.standard_normal(s.arrays[k].shape) * moving[:, None]).astype(np.float32)
    return c


def _batch(count, seed):
    """Scenes of 16 to 2048 bodies (the i-th as large whatever the seed), every tenth with a chain."""
    rng = np.random.default_rng(seed)
    pool = _pool()
    base = [gen.batch_scene(seed * TEMPLATES + i, n_bodies=gen.batch_scene_bodies(i), chain_prob=1.0 if i % 10 == 7 else 0.0,
                            pool=pool) for i in range(min(count, TEMPLATES))]
    return [_with_velocity(base[i % len(base)], rng, 0.5) for i in range(count)]


def _single(case, seed):
    """The scene of a "frame" case, the frames it runs before it is measured and the pairs
    per collider its world has room for (0: the default)."""
    rng = np.random.default_rng(seed)
    if case["scene"] == "mixed":
        return _with_velocity(gen.batch_scene(seed, n_bodies=case["bodies"], chain_prob=0.0, pool=_pool()), rng, 0.5), 30, 16
    if case["scene"] == "pyramid":
        return _with_velocity(gen.pyramid(rows=case["rows"]), rng, 0.01), 8, 0
    if case["scene"] == "terrain":
        s = gen.large_mixed(case["bodies"], cells=case["cells"], seed=gen.scene_seed(2, seed))
        # every column of bodies starts just above the ground under it, so that the lowest have landed
        verts = s.trimesh[0][0].reshape(case["cells"] + 1, case["cells"] + 1, 3)
        pos = s.arrays["pos"]
        i, j = (np.clip(np.rint(pos[1:, k] + case["cells"] / 2), 0, case["cells"]).astype(int) for k in (0, 2))
        pos[1:, 1] += verts[i, j, 1] - (verts[:, :, 1].max() + 6.0) + 1.6
        return s, 20, 16
    return gen.joint_chains(case["chains"], links=case["links"], seed=gen.scene_seed(3, seed)), 10, 16


def _page_locked(state):
    """Page-locked copies of body arrays (torch tensors; numpy views share them)."""
    out = {}
    for k in KEYS:
        out[k] = torch.empty(state[k].shape, dtype=torch.float32, pin_memory=True)
        out[k].copy_(torch.from_numpy(np.ascontiguousarray(state[k])))
    return out


def _held(world, frames):
    """The world after `frames` frames, with its body state in page-locked arrays: the
    state every pass starts from, and the arrays that a frame reads and writes."""
    world.step(frames=frames)
    world.synchronize()
    start = _page_locked(world.read_bodies())
    live = {k: torch.empty_like(v, pin_memory=True) for k, v in start.items()}
    return {"world": world, "start": start, "start_np": {k: v.numpy() for k, v in start.items()}, "live": live,
            "live_np": {k: v.numpy() for k, v in live.items()}, "dt": world.scenes[0].dt}


def _rays(case, seed, ss):
    """Rays from outside each scene's bodies towards points among them."""
    rng = np.random.default_rng(seed + 1)
    n = case["rays"]
    scene = np.sort(rng.integers(0, len(ss), n))
    lo = np.stack([s.arrays["pos"][1:].min(0) for s in ss]).astype(np.float64)
    hi = np.stack([s.arrays["pos"][1:].max(0) for s in ss]).astype(np.float64)
    mid, half = ((lo + hi) / 2)[scene], ((hi - lo) / 2)[scene]
    target = mid + half * rng.uniform(-1.1, 1.1, (n, 3))
    yaw = rng.uniform(0, 2 * math.pi, n)
    reach = np.linalg.norm(half, axis=1) + 6.0
    origin = mid + np.stack([reach * np.cos(yaw), rng.uniform(0.2, 0.8, n) * reach, reach * np.sin(yaw)], 1)
    d = target - origin
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rows = np.zeros((n, 8), np.float32)
    rows[:, 0] = scene
    rows[:, 1:4], rows[:, 4:7], rows[:, 7] = origin, d, 200.0
    return rows


def _ray_scenes(case, seed):
    pool = _pool()
    return [gen.batch_scene(seed * 64 + i, n_bodies=case["bodies"], chain_prob=0.0, pool=pool) for i in range(case["scenes"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        s, frames, ppc = _single(case, seed)
        return dict(_held(World([s], pairs_per_collider=ppc), frames), kind=kind)
    if kind in ("batch", "rollout"):
        w = World(_batch(case["scenes"], seed), use_graph=True)
        return dict(_held(w, 10), kind=kind, frames=case.get("frames", 1))
    if kind == "serve":
        pool = _pool()
        holder = gen.SceneData("hulls")
        holder.convex.extend(pool)
        holder.add_bodies(pos=[[0, 0, 0]], quat=[gen.IDENTITY_Q], flags=0, inv_mass=0.0, com=np.zeros(3),
                          inv_inertia=np.zeros(9), col_type=gen.SPHERE, col_params=[0.5, 0, 0, 0], col_mesh=-1)
        sizes, reqs = np.random.default_rng(case["requests"]), []    # the same requests' sizes for every seed
        for i in range(case["requests"]):
            n = int(round(math.exp(sizes.uniform(math.log(8), math.log(case["max_bodies"])))))
            s = gen.batch_scene(seed * 64 + i, n_bodies=n, config=5, chain_prob=0.0, pool=pool)
            reqs.append((s, int(sizes.integers(1, case["max_frames"] + 1)), make_desc(s)))
        return {"kind": kind, "server": Server(SERVE_CLASSES, mesh_pool=holder.finalize()), "requests": reqs,
                "per_tick": case["per_tick"]}
    if kind == "rays":
        ss = _ray_scenes(case, seed)
        return {"kind": kind, "world": World(ss), "rays": _rays(case, seed, ss)}
    if kind == "characters":
        n = case["scenes"]
        rng = np.random.default_rng(seed)
        base, chars = gen.character_scene(seed=seed, n_chars=1, n_balls=case["balls"])
        w = World([_with_velocity(base, rng, 0.3) for _ in range(n)], use_graph=True)
        specs = [{"scene": i, "body": chars[0], "height": 1.0, "radius": 0.3} for i in range(n)]
        return dict(_held(w, 20), kind=kind, specs=specs, moves=gen.character_moves(n, 1, seed=seed)[0])
    verts, idx, _ = gen.heightfield(gen.SplitMix64(gen.scene_seed(2, seed)), cells=case["cells"])
    return {"kind": kind, "vertices": verts, "indices": idx}


# ---------------------------------------------------------------- one pass

def _serve(state):
    """Admit `per_tick` requests a tick as slots allow, tick until all have run, and read
    each request's final state while the next tick runs."""
    srv, reqs = state["server"], state["requests"]
    nxt, live, done, final = 0, {}, [], [None] * len(reqs)
    while live or done or nxt < len(reqs):
        for _ in range(state["per_tick"]):
            if nxt == len(reqs):
                break
            scene, frames, desc = reqs[nxt]
            slot = srv.admit(scene, frames, desc=desc)
            if slot is None:
                break
            live[slot] = nxt
            nxt += 1
        busy = bool(live)
        if busy:
            srv.tick_begin()
        for slot, r in done:
            final[r] = srv.read(slot)
            srv.release(slot)
        done = [(slot, live.pop(slot)) for slot in srv.tick_end()] if busy else []
    return {k: np.concatenate([f[k] for f in final]) for k in KEYS}


def run(state):
    kind = state["kind"]
    if kind in ("frame", "batch"):
        for k in KEYS:                      # the registry's state of this frame
            state["live"][k].copy_(state["start"][k])
        state["world"].simulate_host(state["dt"], state["live_np"])
        return state["live"]
    if kind == "rollout":
        w = state["world"]
        w.write_bodies(state["start_np"])
        w.step(state["dt"], frames=state["frames"])
        return w.read_bodies()
    if kind == "serve":
        return _serve(state)
    if kind == "rays":
        return state["world"].raycast(state["rays"])
    if kind == "characters":
        w = state["world"]
        w.write_bodies(state["start_np"])
        flags = w.move_characters(state["specs"], state["moves"], state["dt"])
        w.step(state["dt"])
        return dict(w.read_bodies(), flags=flags)
    return list(trimesh_build(state["vertices"], state["indices"]))


# ---------------------------------------------------------------- what a pass cannot do without

BODY_STATE = 52          # position, orientation and two velocities, in bytes
BODY_FIXED = 140         # mass, inertia, collider pose, shape and material
POINTS = 0.8             # contact points per body in the scenes here
ROW_FLOPS = 95           # one contact or joint row solved once


def work(case):
    kind = case["kind"]
    frames, steps, sweeps = case.get("frames", 1), 4, 9
    if kind == "rays":
        n = case["scenes"] * (case["bodies"] + 1)
        return {"bytes": case["rays"] * (32 + 28) + n * 108, "flops": case["rays"] * 30 * (math.log2(case["bodies"] + 1) + 4)}
    if kind == "trimesh":
        t, v = 2 * case["cells"] ** 2, (case["cells"] + 1) ** 2
        return {"bytes": 12 * v + 12 * t + 80 * t + 32 * (2 * t - 1), "flops": 60 * t * math.log2(t)}
    rows = None
    if kind == "frame":
        if case["scene"] == "pyramid":
            n = case["rows"] * (case["rows"] + 1) // 2
            rows = 2 * 4.4 * n
        elif case["scene"] == "chains":
            n, steps, sweeps = case["chains"] * case["links"], 8, 5
            rows = 4.4 * n
        else:
            n = case["bodies"]
    elif kind in ("batch", "rollout"):
        n = case["scenes"] * 413
    elif kind == "serve":
        mean = (case["max_bodies"] - 8) / math.log(case["max_bodies"] / 8)
        n, frames = case["requests"] * mean, (case["max_frames"] + 1) / 2
    else:
        n = case["scenes"] * (case["balls"] + 1)
    rows = 2 * POINTS * n if rows is None else rows
    return {"bytes": n * (2 * BODY_STATE + BODY_FIXED), "flops": frames * steps * (rows * sweeps * ROW_FLOPS + n * 400)}


# ---------------------------------------------------------------- ray queries in 64 bits

def _matrices(q):
    x, y, z, w = (q[:, i] for i in range(4))
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)


def _sphere_hit(o, d, r):
    """Entry distance of rays o + t d (from outside) into spheres of radius r about the origin."""
    b, c = (o * d).sum(-1), (o * o).sum(-1) - r * r
    disc = b * b - c
    t = -b - np.sqrt(np.maximum(disc, 0))
    return np.where((disc >= 0) & (t >= 0), t, np.inf)


def _planes_hit(num, den):
    """Entry distance into the half spaces den * t <= num, all of them."""
    with np.errstate(divide="ignore", invalid="ignore"):
        t = num / den
    enter = np.max(np.where(den < 0, t, -np.inf), -1)
    leave = np.min(np.where(den > 0, t, np.inf), -1)
    clear = np.all((den != 0) | (num >= 0), -1)
    return np.where(clear & (enter <= leave) & (enter >= 0), enter, np.inf)


def exact(case, seed):
    """Closest hits by testing every ray against every collider of its scene."""
    if case["kind"] != "rays" or case["rays"] * case["bodies"] > 4e7:
        return None
    ss = _ray_scenes(case, seed)
    rays = _rays(case, seed, ss)
    scene = rays[:, 0].astype(np.int64)
    dist = np.zeros(len(rays))
    for si, s in enumerate(ss):
        sel = np.nonzero(scene == si)[0]
        o, d = rays[sel, 1:4].astype(np.float64), rays[sel, 4:7].astype(np.float64)
        a = s.arrays
        best = np.full(len(sel), np.inf)
        rot = _matrices(a["quat"].astype(np.float64))
        for b in range(len(a["pos"])):
            lo, ld = (o - a["pos"][b]) @ rot[b], d @ rot[b]       # the ray in the body's frame
            p = a["col_params"][b].astype(np.float64)
            t = a["col_type"][b]
            if t == gen.SPHERE:
                h = _sphere_hit(lo, ld, p[0])
            elif t == gen.CAPSULE:
                hh, r = p[0], p[1]
                h = np.full(len(sel), np.inf)
                for end in (hh, -hh):
                    c = _sphere_hit(lo - [0, end, 0], ld, r)
                    y = lo[:, 1] + np.where(np.isfinite(c), c, 0) * ld[:, 1]
                    h = np.minimum(h, np.where((y >= hh) if end > 0 else (y < -hh), c, np.inf))
                qa, qb = ld[:, 0] ** 2 + ld[:, 2] ** 2, lo[:, 0] * ld[:, 0] + lo[:, 2] * ld[:, 2]
                disc = qb * qb - qa * (lo[:, 0] ** 2 + lo[:, 2] ** 2 - r * r)
                with np.errstate(divide="ignore", invalid="ignore"):
                    c = np.where(disc >= 0, (-qb - np.sqrt(np.maximum(disc, 0))) / qa, np.inf)
                y = lo[:, 1] + np.where(np.isfinite(c), c, 0) * ld[:, 1]
                h = np.minimum(h, np.where((c >= 0) & (y >= -hh) & (y < hh), c, np.inf))
            elif t == gen.BOX:
                h = _planes_hit(np.concatenate([p[:3] - lo, p[:3] + lo], 1), np.concatenate([ld, -ld], 1))
            else:
                m = int(a["col_mesh"][b])
                f0, f1 = a["convex_face_start"][m], a["convex_face_start"][m + 1]
                nrm = a["face_normal"][f0:f1].astype(np.float64) / p[:3]
                cen = a["face_centroid"][f0:f1].astype(np.float64) * p[:3]
                h = _planes_hit((nrm * cen).sum(1) - lo @ nrm.T, ld @ nrm.T)
            best = np.minimum(best, h)
        dist[sel] = best
    hit = dist <= rays[:, 7]
    dist = np.where(hit, dist, 0.0)
    pos = np.where(hit[:, None], rays[:, 1:4].astype(np.float64) + rays[:, 4:7].astype(np.float64) * dist[:, None], 0.0)
    return {"body": None, "collider": None, "entity": None, "distance": dist, "pos": pos}

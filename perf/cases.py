"""The work that programs have this framework do, as cases to be timed.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call, run() is one pass through the public
entry points, work() what a pass cannot do without.

How a program calls the framework, by kind:
  frame   a game's frame: one step (pair list on the device), then the bulk
          state export a renderer reads
  dropin  the engine's own step with the pair list handed across the boundary:
          pairs out, step with pairs in, body records back
  narrow  an engine that keeps its own solver: it moves the bodies, then asks
          for pairs and contact manifolds
  pairs   the broad phase alone, over a whole level
  edit    a destructible terrain: voxels carved or filled, a step, the state
          and the edited voxels read back (the mesh is rebuilt from them)
  stream  a streamed voxel world: some terrain chunks replaced by new ones,
          a step, the state read back
  batch   many independent worlds restarted from a checkpoint, advanced
          together for some steps, every world's bodies read back
  serve   a queue of simulation jobs of uneven sizes drained by the server

Scenes that evolve return to their starting bodies every EPISODE frames, as an
episode or a replayed level does, so that a pass's work does not depend on how
many passes came before it.

No 64-bit values are given (exact): a step chooses its contacts by comparing
and flooring 32-bit positions and then solves thousands of dependent contact
rows one after another.  In 64 bits other contacts can be chosen, so there is no
common value to measure an error against, and in plain numpy the smallest scene
takes longer than the comparison allows.  The pair lists and voxels are whole
numbers.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

vxp = importlib.import_module("zig-voxel-physics_b200")
scenes, abi = vxp.scenes, vxp.abi

EPISODE = 60


def listed():
    return [
        # a menu screen or a puzzle: a handful of crates; launches and latency
        dict(name="frame_5_cubes", kind="frame", shape="cubes", bodies=5, settle=90),
        # the small scene of the benchmark: 64 one-brick cubes on a slab
        dict(name="frame_64_cubes", kind="frame", shape="cubes", bodies=64, settle=100),
        # a room of rubble, just past the size that is stepped by the whole GPU
        dict(name="frame_523_boxes", kind="frame", shape="boxes", bodies=523, settle=240),
        # the benchmark's large pile
        dict(name="frame_4096_boxes", kind="frame", shape="boxes", bodies=4096, settle=360),
        # the engine's drop-in call with host pair lists and body records
        dict(name="dropin_1331_boxes", kind="dropin", shape="boxes", bodies=1331, settle=300),
        # contacts for an engine with its own solver
        dict(name="narrow_900_boxes", kind="narrow", shape="boxes", bodies=900, settle=280),
        # large irregular bodies (64^3 value noise): voxel contact generation
        dict(name="frame_125_noise64", kind="frame", shape="noise", bodies=125, size=64, settle=4),
        # a crater every frame in a 64^3 terrain with cubes on it
        dict(name="edit_64", kind="edit", bodies=61, size=64, radius=4, settle=60),
        # terrain streaming: 4 of 16 chunks of 32^3 replaced each frame
        dict(name="stream_16_chunks", kind="stream", bodies=48, size=32, chunks=16, fresh=4, settle=20),
        # the pair list of a large level
        dict(name="pairs_15000", kind="pairs", shape="boxes", bodies=15000),
        # the batched mix: 256 worlds, sizes log-uniform in 8..2048
        dict(name="batch_256_worlds", kind="batch", worlds=256, lo=8, hi=2048, settle=150, steps=60),
        # the served mix: jobs of 16..4096 bodies, more jobs than slots
        dict(name="serve_40_jobs", kind="serve", jobs=40, slots=24, lo=16, hi=4096, steps_lo=20, steps_hi=90),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cubes", "boxes", "boxes", "noise", "dropin", "narrow", "pairs", "edit", "stream", "batch", "serve"])
    if kind == "cubes":
        return dict(kind="frame", shape="cubes", bodies=logint(1, 500), settle=rng.randint(30, 150),
                    reference=rng.random() < 0.25)
    if kind == "boxes":
        return dict(kind="frame", shape="boxes", bodies=logint(8, 4000), settle=rng.randint(100, 360))
    if kind == "noise":
        return dict(kind="frame", shape="noise", bodies=logint(2, 64), size=rng.randint(17, 64), settle=rng.randint(1, 20))
    if kind in ("dropin", "narrow"):
        return dict(kind=kind, shape="boxes", bodies=logint(8, 2500), settle=rng.randint(100, 360))
    if kind == "pairs":
        return dict(kind="pairs", shape="boxes", bodies=logint(100, 15000))
    if kind == "edit":
        return dict(kind="edit", bodies=logint(1, 200), size=8 * rng.randint(2, 8), radius=rng.randint(1, 6),
                    settle=rng.randint(10, 90))
    if kind == "stream":
        chunks = rng.choice([4, 9, 16])
        return dict(kind="stream", bodies=logint(1, 100), size=8 * rng.randint(2, 4), chunks=chunks,
                    fresh=rng.randint(1, 4), settle=rng.randint(5, 40))
    if kind == "batch":
        lo = logint(4, 64)
        return dict(kind="batch", worlds=logint(4, 200), lo=lo, hi=lo * rng.randint(2, 20), settle=rng.randint(60, 150),
                    steps=rng.randint(10, 60))
    jobs = rng.randint(4, 32)
    return dict(kind="serve", jobs=jobs, slots=rng.randint(2, jobs), lo=16, hi=logint(64, 2000),
                steps_lo=10, steps_hi=rng.randint(20, 80))


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _side(n):
    k = 1
    while k ** 3 < n:
        k += 1
    return k


def _cut(scene, statics, n):
    """The scene with its first n dynamic bodies only."""
    bodies = scene.bodies[: statics + n].copy()
    used = set(int(c) for c in bodies["collider_id"])
    return [c for c in scene.colliders if c.id in used], bodies


def _boxes_or_cubes(case, seed):
    n = case["bodies"]
    if case.get("shape") == "cubes" or case["kind"] in ("edit", "stream"):
        s = scenes.config1(n_side=_side(n), seed=seed)
        return (*_cut(s, 1, n), np.float32(1 / 60), dict(substeps=4))
    s = scenes.config2(n_side=_side(n), seed=seed)
    return (*_cut(s, 2, n), np.float32(1 / 120), dict(substeps=8))


@functools.lru_cache(maxsize=8)
def _bin(n):
    return scenes.walled_bin(n, 16, n)


def _noise_bricks(seed, count, size, empty=True):
    """Per collider the bricks of a size^3 value-noise solid (about half full),
    classified from neighbours; empty: bricks without a voxel are kept."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    grid = torch.rand((count, 1, 9, 9, 9), generator=gen, device="cuda")
    s = torch.nn.functional.interpolate(grid, size=(size,) * 3, mode="trilinear", align_corners=True)[:, 0] >= 0.5
    up = -size % 8
    s = torch.nn.functional.pad(s, (1, 1 + up, 1, 1 + up, 1, 1 + up))  # [collider, z, y, x], one empty voxel around
    c = s[:, 1:-1, 1:-1, 1:-1]
    faces = [s[:, 1:-1, 1:-1, :-2], s[:, 1:-1, 1:-1, 2:], s[:, 1:-1, :-2, 1:-1], s[:, 1:-1, 2:, 1:-1],
             s[:, :-2, 1:-1, 1:-1], s[:, 2:, 1:-1, 1:-1]]
    mask = sum((~f).to(torch.int64) << k for k, f in enumerate(faces))
    vtype = np.array([4, 3, 2, 1, 1, 1, 1], dtype=np.uint8)[[bin(m).count("1") for m in range(64)]]
    byte = torch.from_numpy(scenes.voxel_byte(vtype, scenes.NORMAL_INDEX)).cuda()
    vox = torch.where(c, byte[mask], torch.zeros((), dtype=torch.uint8, device="cuda"))
    b = (size + up) // 8
    vox = vox.view(count, b, 8, b, 8, b, 8).permute(0, 1, 3, 5, 2, 4, 6).reshape(count, b ** 3, 512)
    solid = c.flatten(1).sum(1).cpu().numpy()
    vox = vox.cpu().numpy()
    z, y, x = np.meshgrid(np.arange(b), np.arange(b), np.arange(b), indexing="ij")
    pos = np.stack([x, y, z], axis=-1).reshape(-1, 3)
    out = []
    for v in vox:
        keep = v.any(axis=1) | empty
        br = np.zeros(int(keep.sum()), dtype=abi.BRICK_DTYPE)
        br["pos"], br["voxels"] = pos[keep], v[keep]
        out.append(br)
    return out, solid


def _static(bid, cid, pos):
    b = np.zeros(1, dtype=abi.BODY_DTYPE)
    b["id"], b["body_type"], b["collider_id"], b["is_sleeping"] = bid, abi.BODY_STATIC, cid, 1
    b["position"], b["rotation"] = pos, (0, 0, 0, 1)
    b["friction"], b["restitution"] = 0.6, 0.2
    return b


def _noise_scene(case, seed):
    """Noise bodies on a lattice with 10 % overlap in a walled bin."""
    n, size, vs = case["bodies"], case["size"], 0.1
    side, sp = _side(n), 0.9 * size * 0.1
    bricks, solid = _noise_bricks(seed, n, size, empty=False)
    nb = int(math.ceil((side * sp + size * vs) / vs)) + 8
    cols = [scenes.Collider(0, vs, _bin(nb))] + [scenes.Collider(i + 1, vs, br) for i, br in enumerate(bricks)]
    k = np.arange(n)
    b = np.zeros(n, dtype=abi.BODY_DTYPE)
    b["id"], b["body_type"], b["collider_id"] = k + 2, abi.BODY_DYNAMIC, k + 1
    b["position"] = np.stack([4 * vs + (k % side) * sp, 2 * vs + (k // side ** 2) * sp,
                              4 * vs + (k // side % side) * sp], axis=1)
    b["rotation"] = (0, 0, 0, 1)
    b["inv_mass"] = 1.0 / solid
    inertia = solid * (size * vs) ** 2 / 6.0  # of a cube of that mass
    for d in (0, 4, 8):
        b["inv_inertia_local"][:, d] = 1.0 / inertia
    b["friction"], b["restitution"], b["linear_damping"], b["angular_damping"] = 0.6, 0.2, 0.3, 0.5
    return cols, np.concatenate([_static(1, 0, (0, 0, 0)), b]), np.float32(1 / 60), dict(substeps=4)


@functools.lru_cache(maxsize=1)
def _shapes():
    return scenes.shape_library()


def _log_sizes(rng, n, lo, hi):
    """n sizes spread over the logarithm of [lo, hi], in random order."""
    u = (rng.permutation(n) + 0.5) / n
    return np.floor(lo * ((hi + 1) / lo) ** u).astype(int)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _start(state, cols, bodies, dt, config, settle):
    """A system with the scene loaded and settled; its bodies from there on are
    what an episode starts from."""
    s = vxp.VoxelPhysicsSystem(max_bodies=len(bodies), max_pairs=24 * len(bodies) + 1024, **config)
    for c in cols:
        s.add_collider(c.id, c.voxel_size, c.bricks)
    s.set_bodies(bodies)
    for _ in range(settle):
        s.step(dt)
    state.update(system=s, dt=dt, bodies=s.get_bodies(), frame=0)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(kind=kind)
    if kind in ("frame", "dropin", "narrow", "pairs"):
        cols, bodies, dt, config = (_noise_scene if case["shape"] == "noise" else _boxes_or_cubes)(case, seed)
        if case.get("reference"):
            config.update(colouring=abi.COLOUR_REFERENCE, reference_caps=1)
        if kind == "pairs":
            # the level's boxes at the density of a loose heap
            bodies["position"] *= 0.45
        _start(state, cols, bodies, dt, config, case.get("settle", 0))
        if kind == "pairs":
            state["out"] = np.zeros(64 * len(bodies), dtype=abi.PAIR_DTYPE)
        if kind == "narrow":
            state["out"] = np.zeros(24 * len(bodies), dtype=abi.MANIFOLD_DTYPE)
            # the engine's bodies in the frames to come
            tables = [state["bodies"]]
            for _ in range(7):
                state["system"].step(dt)
                tables.append(state["system"].get_bodies())
            state["tables"] = tables
        return state
    if kind == "edit":
        rng = np.random.default_rng(seed)
        size, vs = case["size"], 0.2
        terrain, _ = _noise_bricks(seed, 1, size)
        cols, bodies, dt, config = _boxes_or_cubes(case, seed)
        cols = [scenes.Collider(0, vs, terrain[0]), *[c for c in cols if c.id != 0]]
        bodies["position"][0] = (-size * vs / 2, -size * vs, -size * vs / 2)
        # spheres that reach the surface, each carved in one frame and filled in the next
        r = case["radius"]
        g = np.stack(np.meshgrid(*[np.arange(-r, r + 1)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
        ball = g[(g ** 2).sum(1) <= r * r]
        spots = []
        for _ in range(8):
            at = rng.integers(0, size, size=3)
            at[1] = size - 1 - rng.integers(0, r + 1)
            c = ball + at
            spots.append(c[((c >= 0) & (c < size)).all(1)].astype(np.int32))
        state["spots"] = spots
        _start(state, cols, bodies, dt, config, case["settle"])
        return state
    if kind == "stream":
        size, vs, n = case["size"], 0.2, case["chunks"]
        side = int(math.isqrt(n))
        cols, bodies, dt, config = _boxes_or_cubes(case, seed)
        chunks, _ = _noise_bricks(seed, 2 * n, size)  # the chunks there now, then the ones to come
        statics = [_static(1 + i, 100 + i, ((i % side - side / 2) * size * vs, -size * vs, (i // side - side / 2) * size * vs))
                   for i in range(n)]
        cubes = bodies[1:]
        cubes["id"] += n
        _start(state, [scenes.Collider(100 + i, vs, chunks[i]) for i in range(n)] + [c for c in cols if c.id != 0],
               np.concatenate([*statics, cubes]), dt, config, case["settle"])
        state.update(chunks=chunks, n=n, fresh=case["fresh"], voxel=vs)
        return state
    rng = np.random.default_rng(seed)
    n = case["worlds"] if kind == "batch" else case["jobs"]
    tables = [scenes.job_bodies(dict(seed=int(rng.integers(2 ** 31)), bodies=int(b)))
              for b in _log_sizes(rng, n, case["lo"], case["hi"])]
    dt = np.float32(1 / 60)
    batch = vxp.VoxelWorldBatch(n if kind == "batch" else case["slots"], substeps=4)
    for c in _shapes():
        batch.add_collider(c.id, c.voxel_size, c.bricks)
    state.update(batch=batch, dt=dt)
    if kind == "batch":
        for w, t in enumerate(tables):
            batch.set_world(w, t)
        batch.step(dt, case["settle"])
        batch.synchronize()
        batch.autotune(dt, 2)
        # the checkpoint the worlds restart from
        state.update(tables=[batch.get_world(w) for w in range(n)], steps=case["steps"])
    else:
        steps = rng.integers(case["steps_lo"], case["steps_hi"] + 1, size=n)
        state.update(tables=tables, steps=[int(x) for x in steps], slots=case["slots"])
    return state


_BODY_OUT = ("id", "is_sleeping", "position", "rotation", "linear_velocity", "angular_velocity", "sleep_timer")


def _fields(table, names):
    return {f: table[f] for f in names}


def _keep(state, found):
    """A list of varying length into the program's own buffer, zeros after it."""
    out = state["out"]
    out[: len(found)] = found
    out[len(found): state.get("found", 0)] = 0
    state["found"] = len(found)
    return out


def run(state):
    kind = state["kind"]
    if kind in ("batch", "serve"):
        return _run_worlds(state)
    s, f = state["system"], state["frame"]
    state["frame"] = f + 1
    if kind == "pairs":
        return _fields(_keep(state, s.pairs()), ("body_a", "body_b"))
    if kind == "narrow":
        s.set_bodies(state["tables"][f % len(state["tables"])])
        pairs = s.pairs()
        s.narrow_phase(pairs)
        m = _keep(state, s.manifolds())
        out = _fields(m, ("body_a_id", "body_b_id", "contact_count", "friction", "restitution"))
        out.update(_fields(m["contacts"], ("point", "normal", "penetration", "local_anchor_a", "local_anchor_b",
                                           "normal_impulse", "tangent_impulse", "feature_id")))
        return out
    if f and f % EPISODE == 0:
        s.set_bodies(state["bodies"])
    if kind == "dropin":
        s.step(state["dt"], s.pairs())
        return _fields(s.get_bodies(), _BODY_OUT)
    if kind == "edit":
        spot = state["spots"][f // 2 % len(state["spots"])]
        s.edit_collider(0, spot, np.full(len(spot), f % 2, dtype=np.uint8), "occupancy")
    if kind == "stream":
        n, k = state["n"], state["fresh"]
        for j in range(k):
            i = (f * k + j) % (2 * n)  # round and round: the new chunks, then the old ones again
            s.add_collider(100 + i % n, state["voxel"], state["chunks"][(i + n) % (2 * n)])
    s.step(state["dt"])
    out = s.export_state()
    if kind == "edit":
        _, bricks = s.read_collider(0)
        out["voxels"] = bricks["voxels"]
    return out


def _run_worlds(state):
    batch, dt = state["batch"], state["dt"]
    if state["kind"] == "batch":
        for w, t in enumerate(state["tables"]):
            batch.set_world(w, t)
        batch.step(dt, state["steps"])
        batch.synchronize()
        done = [batch.get_world(w) for w in range(len(state["tables"]))]
    else:
        jobs = [vxp.server.Job(i, 0.0, t, n) for i, (t, n) in enumerate(zip(state["tables"], state["steps"]))]
        vxp.server.SimulationServer(batch, dt, state["slots"]).run(jobs)
        done = [j.result for j in jobs]
    return _fields(np.concatenate(done), _BODY_OUT)


# ---------------------------------------------------------------------------
# the least a pass can do
# ---------------------------------------------------------------------------
_BODY = 128       # one body record
_CONTACT = 92     # a contact record read as the last frame's and written as this one's
_POINTS = 7.0     # contact points per body in the settled scenes
_ROW_FLOPS = 330  # one point in one velocity sweep: a normal and two friction rows
_VOXEL_FLOPS = 60  # one voxel placed in the other body and its neighbourhood tested


def _step_work(bodies, substeps, points=_POINTS, voxels=64.0):
    """One step: body state read and written, contacts likewise, the sweeps."""
    pts = points * bodies
    return (bodies * 2 * _BODY + pts * 2 * _CONTACT,
            pts * _ROW_FLOPS * 2 * substeps + voxels * _VOXEL_FLOPS * bodies)


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        lo, hi = case["lo"], case["hi"]
        n = case["worlds"] if kind == "batch" else case["jobs"]
        steps = case["steps"] if kind == "batch" else (case["steps_lo"] + case["steps_hi"]) / 2
        mean = (hi - lo) / math.log(hi / lo)
        b, f = _step_work(n * mean, 4, points=2.0)  # most of a column of boxes is still falling
        return {"bytes": steps * b + n * mean * 2 * _BODY, "flops": steps * f}
    n = case["bodies"]
    if kind == "pairs":
        return {"bytes": n * (28 + 24 + 8 + 8 * 6), "flops": n * 400}
    if kind == "narrow":
        pts = _POINTS * n
        return {"bytes": n * (_BODY + 5 * 16) + pts * _CONTACT, "flops": n * 5 * 64 * _VOXEL_FLOPS}
    if case.get("shape") == "noise":
        # the overlap shells between lattice neighbours
        shell = 3 * 0.1 * case["size"] ** 3
        b, f = _step_work(n, 4, points=12.0, voxels=shell)
        return {"bytes": b + n * shell * 2, "flops": f}
    b, f = _step_work(n, 8 if case.get("shape") == "boxes" else 4)
    if kind == "edit":
        b += 2 * case["size"] ** 3 / 2
    if kind == "stream":
        b += case["fresh"] * 2 * case["size"] ** 3
    return {"bytes": b, "flops": f}


def exact(case, seed):
    return None

"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points of ``falling_sand_engine_gb300`` as a
program that embeds the library calls them, and hands back what that program reads:
the cell planes, particle records, textures, masks, files. A host program reads them
into pinned buffers that it keeps (``World.state(out)``, ``Batch.download_all``), so
the copies are part of the pass; ``noalloc`` updates planes that the caller owns on
the device.

The sizes are those of the repository's own workloads (bench.py: the 512 x 512 world,
the 4096 x 2048 world with 1M particles, uneven batches with sides of 128 to 2048,
the large world with 200 rigid boxes, served worlds of 256 and up) and of ordinary
game worlds (1920 x 1080, ragged sizes). Worlds run on from pass to pass as a program's
do. A pass is a pure function of the state that ``prepare`` made and of the passes
before it.

All outputs are whole numbers (cells, fixed-point or bit patterns of amounts, packed
bytes, the particle records' own bytes), so there is no ``exact`` value to compare with:
they have to be equal.
"""
import ctypes as C
import math

import numpy as np
import torch

import falling_sand_engine_gb300 as fse

TEXTURES = (fse.TEX_PIXELS, fse.TEX_EMISSION, fse.TEX_FIRE, fse.TEX_FLOW, fse.TEX_CELLS)
CELL_BYTES = 11  # id, colour, scalar, flags: the cell state of the metric's roofline


def listed():
    return [
        # the plain single world of the smallest workload: one frame of a small game,
        # where the chain of passes through few chunks counts
        {"name": "step_512", "kind": "step", "w": 512, "h": 512, "ticks": 1, "graph": 0, "f32": 0, "particles": 0},
        # a game's frame on a world of ragged size: bodies stamped and read back, the
        # tick with temperatures and fires, the render textures read by the host
        {"name": "frame_998x701", "kind": "frame", "w": 998, "h": 701, "bodies": 24, "fires": 1},
        # the single-world workload with a million free particles, four frames
        {"name": "particles_4096x2048", "kind": "step", "w": 4096, "h": 2048, "ticks": 4, "graph": 0, "f32": 0,
         "particles": 1000000},
        # a full-HD world advanced eight ticks by a captured graph
        {"name": "graph_1920x1080", "kind": "step", "w": 1920, "h": 1080, "ticks": 8, "graph": 1, "f32": 0,
         "particles": 0},
        # worlds of uneven size in one batch, by captured graphs, planes read back whole
        {"name": "batch_64_uneven", "kind": "batch", "worlds": 64, "lo": 128, "hi": 2048, "ticks": 8, "f32": 0},
        # the large world: power-law mix of eight materials, 200 rigid boxes stamped and
        # read back around the tick, their mask exported
        {"name": "objects_8192x8192", "kind": "objects", "w": 8192, "h": 8192, "bodies": 200},
        # served worlds: requests of 1 to 16 ticks queued for resident worlds of mixed size
        {"name": "serve_48", "kind": "serve", "worlds": 48, "lo": 256, "hi": 1024, "requests": 96},
        # an engine that owns all device memory: a tick predicted on its own planes from a
        # snapshot that it keeps
        {"name": "noalloc_4096x2048", "kind": "noalloc", "w": 4096, "h": 2048},
        # parity runs: the reference's own order and its f32 amounts
        {"name": "reference_order_1024x512", "kind": "refstep", "w": 1024, "h": 512, "f32": 1},
        # saving a world as chunk files (encode) and loading one (decode)
        {"name": "pack_4096x2048", "kind": "pack", "w": 4096, "h": 2048},
        {"name": "unpack_4096x2048", "kind": "unpack", "w": 4096, "h": 2048},
        # the conduction step of a world with temperatures, and the temperatures read
        {"name": "temperature_4096x2048", "kind": "temperature", "w": 4096, "h": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "frame", "batch", "objects", "serve", "noalloc", "refstep", "pack",
                       "unpack", "temperature"])
    if kind == "step":
        w, h = _log_int(rng, 200, 4096), _log_int(rng, 200, 2048)
        return {"kind": kind, "w": w, "h": h, "ticks": rng.choice([1, 2, 4]), "graph": rng.choice([0, 1]),
                "f32": rng.choice([0, 0, 1]), "particles": int(w * h * rng.choice([0.0, 0.02, 0.12]))}
    if kind == "frame":
        return {"kind": kind, "w": _log_int(rng, 300, 2048), "h": _log_int(rng, 300, 1200),
                "bodies": rng.randrange(1, 64), "fires": rng.choice([0, 1])}
    if kind == "batch":
        return {"kind": kind, "worlds": _log_int(rng, 4, 64), "lo": 128, "hi": rng.choice([512, 1024, 2048]),
                "ticks": rng.choice([1, 4, 8]), "f32": rng.choice([0, 0, 1])}
    if kind == "objects":
        return {"kind": kind, "w": _log_int(rng, 1024, 8192), "h": _log_int(rng, 1024, 8192),
                "bodies": rng.randrange(50, 201)}
    if kind == "serve":
        return {"kind": kind, "worlds": _log_int(rng, 8, 48), "lo": 256, "hi": rng.choice([512, 1024]),
                "requests": rng.randrange(16, 97)}
    if kind == "noalloc":
        return {"kind": kind, "w": _log_int(rng, 256, 4096), "h": _log_int(rng, 256, 2048)}
    if kind == "refstep":
        return {"kind": kind, "w": _log_int(rng, 256, 1024), "h": _log_int(rng, 128, 512), "f32": rng.choice([0, 1])}
    return {"kind": kind, "w": _log_int(rng, 256, 4096), "h": _log_int(rng, 256, 2048)}


# ------------------------------------------------------------------- inputs
def _materials():
    fse.InitMaterials()
    fse.PushMaterials()


def _pinned(dtype, *shape):
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    return torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy().view(dtype).reshape(shape)


def _planes(w, h):
    """Pinned host planes for World.state(out)."""
    return {k: _pinned(dt, h, w) for k, dt in fse.World.PLANES}


def _signed(planes):
    """The planes as signed arrays of the same bytes (torch has few unsigned operations)."""
    return {k: a.view({2: np.int16, 4: np.int32}.get(a.itemsize, a.dtype)) for k, a in planes.items()}


def _records(cap):
    """A kept buffer for the particle list."""
    r = _pinned(fse.PARTICLE_DTYPE, cap)
    r.view(np.uint8)[:] = 0
    return r


def _read_particles(world, records):
    """The particle list into `records`; (records as bytes, particles read)."""
    n = C.c_int(0)
    st = fse.lib().fse_particles_read(world.h, C.c_void_p(records.ctypes.data), len(records), C.byref(n))
    if st != 0:
        raise RuntimeError("fse_particles_read: %d" % st)
    return {"particles": records.view(np.int32), "particle_count": n.value}


def _particles(n, w, h, seed):
    """Free sand: positions uniform over the world, velocities N(0, 2) cells a tick."""
    rng = np.random.default_rng(seed)
    p = np.zeros(n, fse.PARTICLE_DTYPE)
    p["x"] = rng.uniform(0, w, n)
    p["y"] = rng.uniform(0, h, n)
    p["vx"] = rng.normal(0.0, 2.0, n)
    p["vy"] = rng.normal(0.0, 2.0, n)
    p["ay"] = 0.1
    p["fade_time"] = 60
    p["id"] = fse.material_find("GENERIC_SAND")
    p["colour"] = 0xFFFFFFFF
    return p


def _bodies(n, w, h, seed, rotate):
    rng = np.random.default_rng(seed)
    b = np.zeros(n, fse.BODY_DTYPE)
    b["w"] = rng.integers(8, 65, n)
    b["h"] = rng.integers(8, 65, n)
    b["x"] = rng.uniform(0, w - 64, n)
    b["y"] = rng.uniform(0, h - 64, n)
    a = rng.uniform(0, 2 * np.pi, n) if rotate else np.zeros(n)
    b["sin_a"] = np.sin(a)
    b["cos_a"] = np.cos(a)
    b["id"] = fse.material_find("GENERIC_OBJECT")
    b["colour"] = 0xFF808080
    return b


def _sizes(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    return (rng.integers(lo // 64, hi // 64 + 1, (n, 2)) * 64).tolist()


def _with_fires(world, seed):
    """Small fires and pools of lava in a generated world."""
    rng = np.random.default_rng(seed)
    p = world.state()
    for name, n in (("FIRE", 12), ("LAVA", 6)):
        m = fse.material_find(name)
        info = fse.material_get(m)
        for _ in range(n):
            x, y = int(rng.integers(4, world.width - 12)), int(rng.integers(4, int(world.height * 0.6) - 8))
            s = np.s_[y:y + 6, x:x + 8]
            p["id"][s] = m
            p["colour"][s] = np.uint32(int(info[6]) & 0xFFFFFFFF)
            p["scalar"][s] = int(info[13])
            p["flags"][s] = 0
            p["diff"][s] = 0
    world.upload(p)


def prepare(case, seed):
    _materials()
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("step", "refstep"):
        w, h = case["w"], case["h"]
        n = case.get("particles", 0)
        world = fse.World(w, h, seed=seed, f32_fluid=bool(case["f32"]), reference_order=kind == "refstep",
                          particle_capacity=max(w * h // 4, 2 * n, 65536))
        world.generate(fse.GEN_MIX, seed)
        if n:
            world.addCell(_particles(n, w, h, seed))
        s.update(world=world, out=_planes(w, h), records=_records(max(2 * n, w * h // 8)))
    elif kind == "frame":
        w, h = case["w"], case["h"]
        world = fse.World(w, h, seed=seed, render=True, temperature_step=True)
        world.generate(fse.GEN_MIX, seed)
        if case["fires"]:
            _with_fires(world, seed)
        s.update(world=world, bodies=_bodies(case["bodies"], w, h, seed, True), out=_planes(w, h),
                 records=_records(w * h // 8), textures={t: _pinned(np.uint8, h, w, 4) for t in TEXTURES})
    elif kind == "batch":
        sizes = _sizes(case["worlds"], case["lo"], case["hi"], 4242)  # the mix of sizes is the case's, not the seed's
        worlds = []
        for k, (w, h) in enumerate(sizes):
            world = fse.World(w, h, seed=seed + k, f32_fluid=bool(case["f32"]))
            world.generate(fse.GEN_MIX, seed + k)
            worlds.append(world)
        batch = fse.Batch(worlds)
        batch.prepare_graphs(case["ticks"], case["ticks"])
        s.update(batch=batch, worlds=worlds, out=_pinned(np.uint8, batch.io_layout()[1]))
    elif kind == "objects":
        w, h = case["w"], case["h"]
        world = fse.World(w, h, seed=seed, particle_capacity=w * h // 8)
        world.generate(fse.GEN_ZIPF8, seed)
        s.update(world=world, bodies=_bodies(case["bodies"], w, h, seed, False), out=_planes(w, h),
                 mask=_pinned(np.uint8, (w * h + 7) // 8))
    elif kind == "serve":
        sizes = _sizes(case["worlds"], case["lo"], case["hi"], 4243)
        srv = fse.Server(64 << 30, 256)
        slots = [srv.add_world(w, h, fse.GEN_MIX, seed + k, seed=seed + k) for k, (w, h) in enumerate(sizes)]
        rng = np.random.default_rng(seed)
        work = [(slots[int(k)], int(n)) for k, n in zip(rng.integers(0, len(slots), case["requests"]),
                                                        rng.integers(1, 17, case["requests"]))]
        out = {k: _pinned(dt, sum(w * h for w, h in sizes)) for k, dt in fse.World.PLANES}
        views, at = [], 0
        for w, h in sizes:
            views.append({k: out[k][at:at + w * h].reshape(h, w) for k in out})
            at += w * h
        s.update(srv=srv, slots=slots, work=work, out=out, views=views)
    elif kind == "noalloc":
        w, h = case["w"], case["h"]
        with fse.World(w, h, seed=seed) as world:
            world.generate(fse.GEN_MIX, seed)
            world.step(16)
            host = world.state()
        s["kept"] = [torch.from_numpy(host[k].view(t)).cuda()
                       for k, t in (("id", np.int16), ("colour", np.int32), ("scalar", np.int32), ("flags", np.uint8),
                                    ("diff", np.int32))]
        s.update(seed=seed, cap=65536, planes=[torch.empty_like(p) for p in s["kept"]],
                 spawned=torch.zeros(65536 * fse.PARTICLE_DTYPE.itemsize, dtype=torch.uint8, device="cuda"))
    else:
        w, h = case["w"], case["h"]
        world = fse.World(w, h, seed=seed, temperature=kind == "temperature")
        world.generate(fse.GEN_MIX, seed)
        world.step(16)  # a world that has been played for a while
        s["world"] = world
        if kind == "pack":
            nb, nc = C.c_int64(0), C.c_int(0)
            fse.lib().fse_world_pack_bound(w, h, C.byref(nb), C.byref(nc))
            s.update(file=np.zeros(nb.value, np.uint8), offsets=np.zeros(nc.value + 1, np.int64))
        elif kind == "unpack":
            s["data"], s["offsets"] = (a.copy() for a in world.pack())
            s["out"] = _planes(w, h)
        elif kind == "temperature":
            s["out"] = _pinned(np.int16, h, w)
    return s


# --------------------------------------------------------------------- a pass
def run(s):
    kind, case = s["kind"], s["case"]
    if kind in ("step", "refstep"):
        world = s["world"]
        world.step(case.get("ticks", 1), graph=bool(case.get("graph", 0)))
        return {**_signed(world.state(s["out"])), **_read_particles(world, s["records"])}
    if kind == "frame":
        world, bodies = s["world"], s["bodies"]
        world.object_stamp(bodies)
        world.step(1)
        taken = world.object_readback(bodies)
        moving = world.render_dirty()
        world.render_cells()
        for which, texture in s["textures"].items():
            st = fse.lib().fse_world_render_read(world.h, which, C.c_void_p(texture.ctypes.data))
            if st != 0:
                raise RuntimeError("fse_world_render_read: %d" % st)
        return {**_signed(world.state(s["out"])), **_read_particles(world, s["records"]), "taken": taken,
                "bodies": bodies.view(np.int32).copy(), "moving": moving, "textures": list(s["textures"].values())}
    if kind == "batch":
        batch = s["batch"]
        batch.step(case["ticks"], graph_ticks=case["ticks"])
        batch.download_all(s["out"])
        batch.sync()
        return s["out"]
    if kind == "objects":
        world, bodies = s["world"], s["bodies"]
        world.object_stamp(bodies)
        world.step(1)
        world.object_mask(s["mask"])
        taken = world.object_readback(bodies)
        return {**_signed(world.state(s["out"])), "mask": s["mask"], "taken": taken,
                "bodies": bodies.view(np.int32).copy()}
    if kind == "serve":
        srv = s["srv"]
        for slot, n in s["work"]:
            srv.submit(slot, n)
        left = len(s["work"])
        while left:
            srv.step()
            left -= len(srv.poll()[0])
        for slot, view in zip(s["slots"], s["views"]):
            srv.world(slot).state(view)
        return _signed(s["out"])
    if kind == "noalloc":
        for p, k in zip(s["planes"], s["kept"]):
            p.copy_(k)
        n = C.c_int(0)
        st = fse.lib().fse_tick_noalloc(*(C.c_void_p(p.data_ptr()) for p in s["planes"]), case["w"], case["h"], 128, 3,
                                        s["seed"] & 0xFFFFFFFF, 16, C.c_void_p(s["spawned"].data_ptr()), s["cap"],
                                        C.byref(n), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != 0:
            raise RuntimeError("fse_tick_noalloc: %d" % st)
        return {"planes": s["planes"], "spawned": s["spawned"], "spawned_count": n.value}
    if kind == "pack":
        n = C.c_int(0)
        st = fse.lib().fse_world_pack(s["world"].h, 0, C.c_void_p(s["file"].ctypes.data), s["file"].size,
                                      C.c_void_p(s["offsets"].ctypes.data), C.byref(n))
        if st != 0:
            raise RuntimeError("fse_world_pack: %d" % st)
        return {"file": s["file"], "offsets": s["offsets"], "chunks": n.value}
    if kind == "unpack":
        phases = s["world"].unpack(s["data"], s["offsets"])
        return {"phases": phases, "planes": _signed(s["world"].state(s["out"]))}
    world = s["world"]
    world.tickTemperature()
    return world.temperature(s["out"])


def exact(case, seed):
    """No output is a rounded value: cells, records and bytes are equal or wrong."""
    return None


# ----------------------------------------------------------------------- work
def work(case):
    """Each tick reads and writes the state of its cells and particles once; what the
    host reads is written once more."""
    kind = case["kind"]
    rec = fse.PARTICLE_DTYPE.itemsize
    if kind in ("batch", "serve"):
        sizes = _sizes(case["worlds"], case["lo"], case["hi"], 4242 if kind == "batch" else 4243)
        cells = sum(w * h for w, h in sizes)
        # a served world runs its share of the requests' 1 to 16 ticks
        ticks = case["ticks"] if kind == "batch" else case["requests"] * 8.5 / case["worlds"]
    else:
        cells = case["w"] * case["h"]
        ticks = case.get("ticks", 1)
    tick_bytes = 2.0 * CELL_BYTES * cells * ticks
    read_out = 15.0 * cells
    if kind == "step":
        nbytes = tick_bytes + read_out + 2.0 * rec * case["particles"] * ticks
    elif kind == "frame":
        nbytes = tick_bytes + read_out + 5 * 4.0 * cells
    elif kind == "objects":
        nbytes = tick_bytes + read_out + cells / 8.0
    elif kind == "noalloc":
        nbytes = tick_bytes + 2 * 15.0 * cells  # and the snapshot copied
    elif kind == "pack":
        nbytes = 7.0 * cells + 1.2 * cells  # id, colour and temperature read, the packed chunks written
    elif kind == "unpack":
        nbytes = 1.2 * cells + read_out * 2
    elif kind == "temperature":
        nbytes = 6.0 * cells + 4.0 * cells + 2.0 * cells  # id and scalar read, scalar written, temperatures read out
    else:
        nbytes = tick_bytes + read_out
    return {"bytes": float(nbytes), "flops": 0.0}

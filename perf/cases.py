"""What the chunk generation and meshing library is timed on: the calls a voxel engine makes
through voxgpu's public entry points, over the sizes, generators, layouts and culling modes
that the library takes.

Every output is whole numbers or record bytes (occupancy, faces, offsets, draw records,
pixels), viewed as integers, and is equal bit for bit whatever computes it; there is no
rounded output, so `exact` has no value to give.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "wgpu-voxel-engine_gb300")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import voxgpu  # noqa: E402

VERTEX, INSTANCED = voxgpu.LAYOUT_VERTEX, voxgpu.LAYOUT_INSTANCED
REFERENCE, FULL6 = voxgpu.CULL_REFERENCE, voxgpu.CULL_FULL6

# The generators of the repository's own workloads; the height of rolling terrain follows the
# chunk size, so that chunks of every size are a mix of air, solid and surface.
GENERATORS = {
    "plain": dict(kind=voxgpu.GEN_HEIGHTMAP, octaves=1, frequency=1.0 / 64, amplitude=12.0,
                  base_height=4.0),
    "terrain": dict(kind=voxgpu.GEN_HEIGHTMAP, octaves=4, frequency=1.0 / 128),
    "caves": dict(kind=voxgpu.GEN_DENSITY, octaves=3, frequency=1.0 / 96, y_ref=256.0,
                  y_scale=1.0 / 64),
    "static": dict(kind=voxgpu.GEN_BERNOULLI),
}
# Arithmetic of one sample: per octave, a 2-D or 3-D Perlin evaluation and its fBm step.
FLOPS = {"plain": 47, "terrain": 47, "caves": 98, "static": 0}
# Mean faces of a chunk over N^2, by chunk size (reference culling emits every face on the
# y borders; so do worlds one layer high).
FACES = {("plain", REFERENCE): {8: 2.0, 16: 2.1, 32: 2.1, 64: 2.1},
         ("terrain", REFERENCE): {8: 1.6, 16: 1.9, 32: 2.3, 64: 3.3},
         ("caves", REFERENCE): {8: 1.3, 16: 1.6, 32: 1.4, 64: 2.1},
         ("caves", FULL6): {8: 0.35, 16: 0.6, 32: 0.7, 64: 1.35}}


def listed():
    return [
        # one chunk remeshed after an edit or a new neighbour: Chunk::create_mesh
        dict(name="one chunk", op="mesh", size=32, gen="caves", n=1, layout=VERTEX, cull=REFERENCE),
        # what a streaming tick dispatches at walking speed: a few chunks on the edge of view
        dict(name="stream tick", op="batch", size=16, gen="terrain", n=3, layout=VERTEX,
             cull=REFERENCE),
        # the 8 x 8 start world at the engine's chunk size, in the renderer's instance layout
        dict(name="start world", op="batch", size=32, gen="plain", n=64, layout=INSTANCED,
             cull=REFERENCE),
        # a world of small terrain chunks refilled by one tuned, captured launch
        dict(name="terrain world", op="graph", size=16, gen="terrain", n=1024, layout=VERTEX,
             cull=REFERENCE),
        # caves and overhangs, very uneven chunks, tuned and captured
        dict(name="cave world", op="graph", size=32, gen="caves", n=4096, layout=VERTEX,
             cull=REFERENCE),
        # the most faces a world can have, bound by the output
        dict(name="densest world", op="graph", size=64, gen="static", n=512, layout=VERTEX,
             cull=REFERENCE),
        # neighbour rebuilds from resident occupancy, culled on all six sides
        dict(name="rebuild", op="rebuild", size=32, gen="caves", n=777, layout=VERTEX, cull=FULL6),
        # meshes delivered into host buffers that a renderer uploads
        dict(name="host meshes", op="host", size=16, gen="terrain", n=1024, layout=VERTEX,
             cull=REFERENCE),
        # Chunk::new for many chunks: one byte per voxel for code that reads cubes
        dict(name="new chunks", op="cubes", size=32, gen="terrain", n=1500, layout=VERTEX,
             cull=REFERENCE),
        # edited or loaded cubes packed back to occupancy
        dict(name="loaded cubes", op="pack", size=32, gen="caves", n=2048, layout=VERTEX,
             cull=REFERENCE),
        # one frame over the view disk of radius 24: visibility and the draw list
        dict(name="frame", op="frame", size=16, gen="terrain", n=1809, layout=VERTEX,
             cull=REFERENCE),
        # a headless 720p image of the start world
        dict(name="image", op="image", size=32, gen="plain", n=64, layout=VERTEX, cull=REFERENCE,
             width=1280, height=720),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["mesh", "batch", "batch", "graph", "graph", "rebuild", "host", "cubes", "pack",
                     "frame", "image"])
    size = rng.choice([8, 16, 16, 32, 32, 64])
    gen = rng.choice(["plain", "terrain", "caves", "caves"])
    case = dict(op=op, size=size, gen=gen, n=1, layout=rng.choice([VERTEX, VERTEX, INSTANCED]),
                cull=rng.choice([REFERENCE, REFERENCE, FULL6]))
    most = {8: 16384, 16: 8192, 32: 4096, 64: 512}[size]
    if op in ("batch", "rebuild"):
        case["n"] = _spread(rng, 1, most // 2)
    elif op == "graph":
        if size == 64 and rng.random() < 0.5:
            case["gen"] = "static"
        case["n"] = _spread(rng, 32, most)
    elif op == "host":
        case["n"] = _spread(rng, 1, {8: 4096, 16: 2048, 32: 512, 64: 64}[size])
    elif op in ("cubes", "pack"):
        case["n"] = _spread(rng, 1, {8: 65536, 16: 16384, 32: 4096, 64: 512}[size])
    elif op == "frame":
        case["n"] = _spread(rng, 50, 50000)
    elif op == "image":
        case["size"] = rng.choice([16, 32])
        case["gen"] = rng.choice(["plain", "terrain"])
        case["layout"] = VERTEX
        case["n"] = _spread(rng, 16, 256)
        case["width"] = _spread(rng, 160, 3840)
        case["height"] = max(90, case["width"] * 9 // 16 + rng.randrange(-3, 4))
    return case


def _config(case, seed):
    size = case["size"]
    gen = dict(GENERATORS[case["gen"]], seed=1 + seed % 1000003)
    if case["gen"] == "terrain":
        gen.update(amplitude=3.0 * size, base_height=size / 2.0)
    return voxgpu.make_config(chunk_size=size, layout=case["layout"], cull_mode=case["cull"],
                              lacunarity=2.0, gain=0.5, **gen)


def _coords(case, rng):
    """n chunks around a place of the world: a patch of ground, or a block around the cave
    layer; the last row of an odd count is ragged."""
    n, size = case["n"], case["size"]
    if case["gen"] == "static":
        return [(i, 0, 0) for i in range(n)]
    cx, cz = rng.randrange(-2000, 2000), rng.randrange(-2000, 2000)
    if case["gen"] == "caves":
        side = max(1, math.ceil(n ** (1.0 / 3.0) - 1e-9))
        mid = 256 // size
        ys = range(mid - side // 2, mid - side // 2 + side)
    else:
        side = max(1, math.ceil(math.sqrt(n)))
        ys = [0]
    return voxgpu.grid_coords(range(cx, cx + side), ys, range(cz, cz + side))[:n]


def _context(cfg):
    # the caller's stream: torch's default stream is CUDA's legacy stream (handle 1)
    return voxgpu.Context(cfg, stream=torch.cuda.current_stream().cuda_stream or 1)


def _device(values, dtype):
    return torch.from_numpy(np.ascontiguousarray(values, dtype=dtype)).cuda()


def _bytes(count):
    return torch.zeros((count + 31) // 16 * 16, dtype=torch.uint8, device="cuda")


def _room(case):
    """Faces that a caller makes room for: well above what such chunks have."""
    if case["gen"] == "static":
        return int(_face_count(case) * 1.01) + 4096
    return 6 * case["size"] ** 2 * case["n"]


class _Meshes:
    """Output buffers of a meshing call, and what the call writes into them."""

    def __init__(self, case, sizes, make=_bytes):
        self.room = _room(case)
        self.offsets = make(8 * (case["n"] + 1))[:8 * (case["n"] + 1)].view(torch.int64)
        self.out0 = make(self.room * sizes.bytes_per_face_out0)
        self.out1 = make(self.room * sizes.bytes_per_face_out1) if sizes.bytes_per_face_out1 else None

    def outputs(self):
        out = [self.offsets, self.out0.view(torch.int64)]
        return out + ([self.out1.view(torch.int64)] if self.out1 is not None else [])


def _pinned(count):
    return torch.zeros((count + 31) // 16 * 16, dtype=torch.uint8, pin_memory=True)


def _neighbour_slots(coords, full6):
    at = {c: i for i, c in enumerate(coords)}
    steps = [(-1, 0, 0), (1, 0, 0), (0, 0, -1), (0, 0, 1), (0, -1, 0), (0, 1, 0)]
    return [[at.get((x + dx, y + dy, z + dz), -1) if k < 4 or full6 else -1
             for k, (dx, dy, dz) in enumerate(steps)] for (x, y, z) in coords]


def _camera(rng, size, eye):
    yaw = rng.uniform(0.0, 2.0 * math.pi)
    look = (math.cos(yaw) * 0.94, -0.34, math.sin(yaw) * 0.94)
    return voxgpu.camera_matrix(eye, look, zfar=1000.0)


def _disk(case, rng):
    """The n chunks nearest to a place, in the order a view disk is walked."""
    radius = math.ceil(math.sqrt(case["n"] / math.pi)) + 1
    cx, cz = rng.randrange(-2000, 2000), rng.randrange(-2000, 2000)
    near = sorted(((dx * dx + dz * dz, dz, dx) for dz in range(-radius, radius + 1)
                   for dx in range(-radius, radius + 1)))[:case["n"]]
    return (cx, cz), sorted((cx + dx, 0, cz + dz) for _, dz, dx in near)


def _place(case, rng, ctx):
    """Coordinates, masks and index base of chunks that have a surface somewhere and fit the
    room made for them (places in open air or deep rock are not what is asked for)."""
    n, full6 = case["n"], case["cull"] == FULL6
    offsets = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    for _ in range(64):
        coords, base = _coords(case, rng), rng.randrange(1 << 20)
        if case["gen"] == "static":
            return coords, None, None, base
        if case["op"] == "batch" and n <= 16:
            # chunks of a streaming tick lie apart on the edge of view; every neighbour counts
            coords = [(x + 37 * i, y, z - 53 * i) for i, (x, y, z) in enumerate(coords)]
            masks = [63 if full6 else 15] * n
        else:
            masks = voxgpu.neighbour_masks(coords, full6)
        c, m = _device(coords, np.int32), _device(masks, np.uint8)
        torch.cuda.synchronize()
        ctx.gen_mesh_batch(c, m, n, None, None, 0, offsets)
        ctx.sync(raise_on_error=False)
        if case["size"] ** 2 <= int(offsets[n]) <= _room(case):
            break
    return coords, c, m, base


def prepare(case, seed):
    rng = random.Random(seed)
    ctx = _context(_config(case, seed))
    full6 = case["cull"] == FULL6
    op, n, size = case["op"], case["n"], case["size"]
    words = ctx.sizes.occ_words_per_chunk
    state = dict(op=op, n=n, ctx=ctx)

    if op == "frame":
        (cx, cz), coords = _disk(case, rng)
        eye = (cx * size + size / 2.0, 60.0, cz * size + size / 2.0)
        np_rng = np.random.RandomState(seed % (1 << 31))
        faces = np_rng.randint(size * size, 4 * size * size, n) * (np_rng.rand(n) < 0.75)
        offsets = np.concatenate([[0], np.cumsum(faces)])
        state.update(coords=_device(coords, np.int32), offsets=_device(offsets, np.int64),
                     planes=voxgpu.frustum_planes(_camera(rng, size, eye)),
                     visible=torch.zeros(n, dtype=torch.uint8, device="cuda"),
                     draws=torch.zeros((n, 5), dtype=torch.int32, device="cuda"),
                     count=torch.zeros(1, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
        return state

    coords, c, masks, base = _place(case, rng, ctx)
    if c is None:
        c = _device(coords, np.int32)
    state.update(coords=c, masks=masks, base=base)
    if op in ("mesh", "batch", "graph", "rebuild", "image"):
        m = state["meshes"] = _Meshes(case, ctx.sizes)
    if op == "mesh":  # one resident chunk with its loaded neighbours
        x, y, z = coords[0]
        around = [(x, y, z), (x - 1, y, z), (x + 1, y, z), (x, y, z - 1), (x, y, z + 1),
                  (x, y - 1, z), (x, y + 1, z)]
        occ = torch.zeros((7, words), dtype=torch.int32, device="cuda")
        c7 = _device(around, np.int32)
        torch.cuda.synchronize()
        ctx.generate(c7, 7, occ)
        state.update(occ=occ, nbrs=[occ[1 + d] if d < 4 or full6 else None for d in range(6)],
                     coord=coords[0], count=torch.zeros(1, dtype=torch.int64, device="cuda"))
    elif op == "graph":
        torch.cuda.synchronize()
        ctx.autotune(c, masks, n, m.out0, m.out1, m.room, m.offsets, chunk_index_base=base)
        state["graph"] = ctx.capture_graph(c, masks, n, m.out0, m.out1, m.room, m.offsets,
                                           chunk_index_base=base)
    elif op == "host":
        state.update(coords=c.cpu().pin_memory(), meshes=_Meshes(case, ctx.sizes, _pinned),
                     masks=masks.cpu().pin_memory())
    elif op in ("rebuild", "cubes", "pack"):
        occ = state["occ"] = torch.zeros((n, words), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        if op != "cubes":
            ctx.generate(c, n, occ)
        if op == "rebuild":
            state.update(slots=torch.arange(n, dtype=torch.int32, device="cuda"),
                         nbrs=_device(_neighbour_slots(coords, full6), np.int32))
        else:
            cubes = state["cubes"] = torch.zeros(n * size ** 3, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            if op == "pack":
                ctx.occ_to_cubes(occ, n, cubes)
    elif op == "image":
        torch.cuda.synchronize()
        ctx.gen_mesh_batch(c, masks, n, m.out0, m.out1, m.room, m.offsets)
        ctx.sync()
        mid = coords[n // 2]
        eye = (mid[0] * size + 0.5, 1.5 * size, mid[2] * size + 0.5)
        width, height = case["width"], case["height"]
        state.update(faces=int(m.offsets[n]), width=width, height=height,
                     view=(ctypes.c_float * 16)(*_camera(rng, size, eye)),
                     keys=torch.zeros(width * height, dtype=torch.int64, device="cuda"),
                     rgba=torch.zeros(width * height, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return state


def run(state):
    op, n, ctx, m = state["op"], state["n"], state["ctx"], state.get("meshes")
    if op == "mesh":
        ctx.mesh(state["occ"][0], state["nbrs"], state["coord"], m.out0, m.out1, m.room,
                 state["count"])
        return [state["count"]] + m.outputs()[1:]
    if op == "batch":
        ctx.gen_mesh_batch(state["coords"], state["masks"], n, m.out0, m.out1, m.room, m.offsets,
                           chunk_index_base=state["base"])
        return m.outputs()
    if op == "graph":
        state["graph"].launch()
        return m.outputs()
    if op == "rebuild":
        ctx.mesh_batch(state["occ"], n, state["slots"], state["nbrs"], state["coords"], n, m.out0,
                       m.out1, m.room, m.offsets)
        return m.outputs()
    if op == "host":
        ctx.gen_mesh_host(state["coords"], state["masks"], n, m.out0, m.out1, m.room, m.offsets,
                          chunk_index_base=state["base"])
        return m.outputs()
    if op == "cubes":
        ctx.generate(state["coords"], n, state["occ"])
        ctx.occ_to_cubes(state["occ"], n, state["cubes"])
        return [state["occ"], state["cubes"]]
    if op == "pack":
        ctx.cubes_to_occ(state["cubes"], n, state["occ"])
        return [state["occ"]]
    if op == "frame":
        ctx.frustum_cull(state["planes"], state["coords"], n, state["visible"])
        ctx.draw_list(state["planes"], state["coords"], state["offsets"], n, state["draws"],
                      state["count"])
        return [state["visible"], state["draws"], state["count"]]
    status = voxgpu.lib().vox_raster(
        ctx._h, ctypes.addressof(state["view"]), m.out0.data_ptr(), m.out1.data_ptr(),
        state["faces"], state["width"], state["height"], state["keys"].data_ptr(),
        state["rgba"].data_ptr())
    if status != voxgpu.VOX_OK:
        raise voxgpu.VoxError(status, "vox_raster")
    return [state["rgba"]]


def _face_count(case):
    size = case["size"]
    if case["gen"] == "static":  # each of the voxel pairs, and each border voxel, with odds 1/2
        per = (3 * size * size * (size - 1) + 6 * size * size) / 2
    else:
        cull = case["cull"] if case["gen"] == "caves" else REFERENCE
        per = FACES[case["gen"], cull][size] * size * size
    return per * case["n"]


def work(case):
    op, n, size, gen = case["op"], case["n"], case["size"], case["gen"]
    face = 120 if case["layout"] == VERTEX else 68
    voxels = n * size ** 3
    octaves = GENERATORS[gen].get("octaves", 0)
    samples = voxels if gen == "caves" else n * size * size  # caves are sampled in 3-D
    noise = samples * octaves * FLOPS[gen]
    if op in ("batch", "graph", "host"):
        return {"bytes": _face_count(case) * face + 13 * n + 8 * (n + 1), "flops": noise}
    if op in ("mesh", "rebuild"):
        halo = 6 if case["cull"] == FULL6 else 4
        read = voxels / 8 + (halo * size * size / 8 if op == "mesh" else 40 * n)
        return {"bytes": _face_count(case) * face + read + 8 * (n + 1), "flops": 0}
    if op == "cubes":
        return {"bytes": voxels + voxels / 8 + 12 * n, "flops": noise}
    if op == "pack":
        return {"bytes": voxels + voxels / 8, "flops": 0}
    if op == "frame":
        return {"bytes": 41 * n, "flops": 2 * n * 8 * 6 * 7}
    return {"bytes": _face_count(case) * 120 + 4 * case["width"] * case["height"],
            "flops": _face_count(case) * 4 * 28}


def exact(case, seed):
    """Every output is whole numbers or record bytes: nothing is rounded."""
    return None

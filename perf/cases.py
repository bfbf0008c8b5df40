"""The calls whose speed matters to a user of the framework, as measurable cases.

Each case is one call (or one edit: two calls) through the public entry points
of leven_gb300, on inputs of the kind the engine makes: chunks around the
terrain surface, the clipmap of a camera, its seams and its meshes, the density
surrogate.  Chunk lists, camera positions, meshes and samples follow from the
seed; the world itself (noise seed, density, the stored CSG operations) is the
same for every seed of a case, as it is in a running engine.

kinds
  chunk   one generateChunkMesh call (no cache), host arrays
  edit    one player edit: applyCSGOperations on a cached chunk, freeChunkOctree, then its new mesh
  tiles   a block of LOD0 chunks around the surface, one batch
  clipmap the nodes nearest a travelling camera, LOD 0 and up, one batch
  frame   all the clipmap nodes of one camera, one batch
  select  clipmap node selection for a set of cameras
  seams   the seam meshes of one camera's clipmap
  collapse  the engine's edge-collapse simplification of a frame's meshes
  train   Adam steps of the density surrogate
  eval    surrogate densities on field lattices
"""
import ctypes as C
import math

import numpy as np
import torch

import leven_gb300 as lvn
from leven_gb300 import workloads as W

DENSITY = {"terrain": dict(mode=lvn.LVN_DENSITY_REFERENCE), "fbm2d": W.FBM2D, "caves": W.CAVES}
ROOT_MIN, ROOT_SIZE = W.CLIPMAP_ROOT_MIN, W.CLIPMAP_ROOT_SIZE
DOMAIN = ((-1024.0, -128.0, -1024.0), (1024.0, 128.0, 1024.0))  # of the surrogate, density units


def listed():
    return [
        # one small chunk of the engine's own terrain, into host arrays: latency
        dict(name="chunk-16-terrain", kind="chunk", vpc=16, scale=1, density="terrain"),
        # the engine's ordinary call: one 64^3 chunk of its own terrain, into host arrays
        dict(name="chunk-64-terrain", kind="chunk", vpc=64, scale=1, density="terrain"),
        # a player's edit of one chunk: dig or fill a sphere, then remesh the cached field
        dict(name="edit-64-fbm2d", kind="edit", vpc=64, scale=1, density="fbm2d", radius=7.5),
        # the block of chunks around a player with stored edits, meshes left on the device
        dict(name="tiles-128-csg", kind="tiles", vpc=64, nx=8, ny=2, nz=8, ops=128, density="fbm2d", memory="device",
             simplify=-1.0),
        # everything a camera sees, of the engine's terrain, into pinned host arrays (a level load)
        dict(name="frame-terrain-pinned", kind="frame", vpc=64, density="terrain", memory="pinned", simplify=-1.0),
        # a streaming batch with caves, simplified for rendering, LOD 0-4
        dict(name="clipmap-1024-simplified", kind="clipmap", vpc=64, n=1024, max_lod=4, ops=0, density="caves",
             memory="device", simplify=0.05),
        # the large sweep: LOD 0-5, caves, stored edits
        dict(name="clipmap-4096-caves", kind="clipmap", vpc=64, n=4096, max_lod=5, ops=64, density="caves",
             memory="device", simplify=-1.0),
        # node selection for the cameras of many views or path positions, lists left on the device
        dict(name="select-4096", kind="select", cameras=4096, memory="device"),
        # the seam meshes that close a whole frame
        dict(name="seams-frame-64", kind="seams", vpc=64, density="caves"),
        # the engine's simplifier on the meshes around the camera
        dict(name="collapse-24", kind="collapse", vpc=64, meshes=24, density="caves"),
        # surrogate training at its usual batch
        dict(name="train-65536", kind="train", steps=32, batch=65536, density="caves"),
        # surrogate fields of a batch's chunks
        dict(name="eval-lattices-32", kind="eval", lattices=32, dim=66, step=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chunk", "chunk", "edit", "tiles", "tiles", "clipmap", "clipmap", "clipmap", "frame", "select",
                       "seams", "collapse", "train", "eval"])
    density = rng.choice(["terrain", "fbm2d", "caves"])
    memory = rng.choice(["device", "device", "pinned"])
    simplify = rng.choice([-1.0, -1.0, round(rng.uniform(0.01, 0.2), 3)])
    if kind == "chunk":
        return dict(kind=kind, vpc=rng.choice([8, 16, 32, 64, 64]), scale=2 ** rng.randint(0, 5), density=density)
    if kind == "edit":
        return dict(kind=kind, vpc=rng.choice([16, 32, 64, 64]), scale=1, density=density,
                    radius=round(rng.uniform(2.0, 12.0), 2))
    if kind == "tiles":
        vpc = rng.choice([16, 32, 64, 64])
        return dict(kind=kind, vpc=vpc, nx=rng.randint(1, 12), ny=rng.randint(1, 3), nz=rng.randint(1, 12),
                    ops=rng.choice([0, _log(rng, 4, 256)]), density=rng.choice(["fbm2d", "fbm2d", "caves"]),
                    memory=memory, simplify=simplify)
    if kind == "clipmap":
        return dict(kind=kind, vpc=64, n=_log(rng, 4, 2048), max_lod=rng.randint(0, 5),
                    ops=rng.choice([0, rng.randint(1, 64)]), density=rng.choice(["fbm2d", "caves", "caves"]),
                    memory=memory, simplify=simplify)
    if kind == "frame":
        return dict(kind=kind, vpc=rng.choice([16, 32, 64]), density=density, memory=memory, simplify=simplify)
    if kind == "select":
        return dict(kind=kind, cameras=_log(rng, 1, 4096), memory=rng.choice(["device", "host"]))
    if kind == "seams":
        return dict(kind=kind, vpc=rng.choice([16, 32, 64]), density=rng.choice(["fbm2d", "caves"]))
    if kind == "collapse":
        return dict(kind=kind, vpc=rng.choice([32, 64]), meshes=rng.randint(1, 24),
                    density=rng.choice(["fbm2d", "caves"]))
    if kind == "train":
        return dict(kind=kind, steps=rng.randint(4, 64), batch=128 * _log(rng, 8, 512),
                    density=rng.choice(["fbm2d", "caves"]))
    dim = rng.choice([18, 34, 66])
    return dict(kind=kind, lattices=_log(rng, 1, 32 if dim == 66 else 256), dim=dim, step=rng.randint(1, 2))


# ---- the world -----------------------------------------------------------------

_ready = False
_probes = {}


def _world(density, ops=()):
    """Noise seed 1, the case's density, and the stored operations."""
    global _ready
    if not _ready:
        lvn.initialise(1, 0, 2)
        _ready = True
    lvn.set_density(**DENSITY[density])
    lvn.clear_csg_operations()
    for op in ops:
        lvn.store_csg_operation(lvn.make_op(op.type, op.brush_shape, op.material, op.origin, op.dimensions, op.rotate_y))


def _context(vpc, simplify=-1.0, cache=0):
    mg = lvn.MeshGen(vpc)
    mg.set_option(lvn.LVN_OPT_CACHE, cache)
    if simplify >= 0.0:
        mg.set_simplify(simplify)
    return mg


def _surface_chunk(density, vpc, scale, seed):
    """The chunk with the most triangles of a column of chunks at a place the seed picks."""
    rng = W.MT19937(seed + 17)
    size = 4 * vpc * scale
    lo, hi = (0, 4000) if density == "terrain" else (-400, 400)  # world units the surface lies in
    x, z = (int(math.floor(rng.uniform(-4096.0, 4096.0) / size)) * size for _ in range(2))
    ys = range(lo // size * size, hi, size)
    chunks = [((x, y, z), size) for y in ys]
    if vpc not in _probes:
        _probes[vpc] = _context(vpc)
    _, _, _, res = _probes[vpc].generate_chunks(chunks)
    return chunks[int(np.argmax(res[:, 3]))]


def _tiles(case, seed):
    """nx x ny x nz chunks, y centred on 0, somewhere in a world with edits over 16 x 16 chunks."""
    rng = W.MT19937(seed + 29)
    v = case["vpc"]
    i0, k0 = (int(rng.uniform(0.0, 16.99 - min(16, case[a]))) for a in ("nx", "nz"))
    y0 = -(4 * v * case["ny"]) // 2
    return [((4 * v * (i0 + i), y0 + 4 * v * j, 4 * v * (k0 + k)), 4 * v)
            for k in range(case["nz"]) for j in range(case["ny"]) for i in range(case["nx"])]


def _camera(rng):
    return [rng.uniform(-1024.0, 1024.0), rng.uniform(-64.0, 64.0), rng.uniform(-1024.0, 1024.0)]


def _clipmap(n, max_lod, seed):
    """The n nodes (LOD 0..max_lod) nearest a camera, of the nodes it has active while it travels."""
    rng = W.MT19937(seed + 43)
    cam = np.array(_camera(rng), np.float64)
    ang, length = rng.uniform(0.0, 2 * math.pi), rng.uniform(160.0, 256.0)
    step = np.array([math.cos(ang) * length, 0.0, math.sin(ang) * length])
    nodes = np.zeros((0, 4), np.int32)
    for k in range(0, 2048, 32):
        cams = cam + np.arange(k, k + 32)[:, None] * step
        got = np.concatenate(lvn.clipmap_select(cams.astype(np.float32), ROOT_MIN, ROOT_SIZE))
        got = got[got[:, 3] <= W.CLIPMAP_LEAF_SIZE << max_lod]
        nodes = np.unique(np.concatenate([nodes, got]), axis=0)
        if len(nodes) >= n or np.abs(cams[-1]).max() > ROOT_SIZE // 2:
            break
    lo, hi = nodes[:, :3].astype(np.float64), nodes[:, :3] + nodes[:, 3:].astype(np.float64)
    d = np.maximum(np.maximum(lo - cam, cam - hi), 0.0)
    order = np.lexsort((nodes[:, 2], nodes[:, 1], nodes[:, 0], nodes[:, 3], (d * d).sum(1)))[:n]
    return [((int(a), int(b), int(c)), int(s)) for a, b, c, s in nodes[order]]


def _frame(seed):
    """All nodes one camera has active, nearest first."""
    cam = np.array([_camera(W.MT19937(seed + 43))], np.float32)
    nodes = lvn.clipmap_select(cam, ROOT_MIN, ROOT_SIZE)[0]
    d = np.abs(nodes[:, :3] + nodes[:, 3:] / 2.0 - cam).max(1)
    return [((int(a), int(b), int(c)), int(s)) for a, b, c, s in nodes[np.argsort(d, kind="stable")]]


def _descs(chunks):
    descs = (lvn.ChunkDesc * len(chunks))()
    for i, (mn, size) in enumerate(chunks):
        descs[i] = lvn.ChunkDesc((C.c_int32 * 3)(*mn), size)
    return descs


def _buffer(shape, dtype, memory):
    """An output buffer; zeroed, so that the part past a mesh's end is the same each time."""
    if memory == "device":
        return torch.zeros(shape, dtype=dtype, device="cuda")
    return torch.zeros(shape, dtype=dtype, pin_memory=memory == "pinned")


FRAME_MAX = 640  # nodes one camera has active: about 430


def _rows(results, n):
    return np.ctypeslib.as_array(C.cast(results, C.POINTER(C.c_int32)), shape=(n, 8))


def _batch_ops(case):
    if case["kind"] == "tiles" and case["ops"]:
        v, h = case["vpc"], case["vpc"] * case["ny"] / 2.0
        return W.csg_ops(case["ops"], 1, (0.0, -h, 0.0), (16.0 * v, h, 16.0 * v))
    if case.get("ops"):
        return W.csg_ops(case["ops"], 1001, (-512.0, -48.0, -512.0), (512.0, 48.0, 512.0))
    return []


# ---- prepare -------------------------------------------------------------------


def _prepare_batch(case, seed):
    _world(case["density"], _batch_ops(case))
    if case["kind"] == "tiles":
        chunks = _tiles(case, seed)
    elif case["kind"] == "clipmap":
        chunks = _clipmap(case["n"], case["max_lod"], seed)
    else:
        chunks = _frame(seed)
    n, f = len(chunks), (case["vpc"] / 64.0) ** 2
    most = {"tiles": n, "clipmap": case.get("n"), "frame": FRAME_MAX}[case["kind"]]
    cap_v, cap_s = int(5000 * f * most) + 262144, int(1024 * f * most) + 65536
    mem = case["memory"]
    s = {"mg": _context(case["vpc"], case["simplify"]), "n": n, "descs": _descs(chunks), "rows": most,
         "results": (lvn.ChunkResult * most)(), "v": _buffer((cap_v, 12), torch.float32, mem),
         "t": _buffer((2 * cap_v, 3), torch.int32, mem), "s": _buffer((cap_s, 12), torch.int32, mem)}
    s["out"] = lvn.BatchOut(lvn.LVN_MEMORY_HOST if mem == "pinned" else lvn.LVN_MEMORY_DEVICE, s["v"].data_ptr(), cap_v,
                            0, s["t"].data_ptr(), 2 * cap_v, 0, s["s"].data_ptr(), cap_s, 0,
                            C.cast(s["results"], C.POINTER(lvn.ChunkResult)))
    return s


def _meshes(vpc, density, seed):
    """One frame meshed on the GPU, as the engine has it before seams and simplification."""
    _world(density)
    chunks = _frame(seed)
    if vpc not in _probes:
        _probes[vpc] = _context(vpc)
    return chunks, _probes[vpc].generate_chunks(chunks)


def _prepare_seams(case, seed):
    chunks, (_, _, S, res) = _meshes(case["vpc"], case["density"], seed)
    rows = np.concatenate([S[o:o + k] for o, k in zip(res[:, 4], res[:, 5])]).astype(np.int32)
    n = len(chunks)
    s = {"n": n, "descs": _descs(chunks), "offs": np.concatenate([[0], np.cumsum(res[:, 5])]).astype(np.int32),
         "rows": torch.from_numpy(rows).cuda(), "vpc": case["vpc"], "hosts": np.arange(n, dtype=np.int32),
         "results": (lvn.ChunkResult * FRAME_MAX)(), "rmin": lvn._ivec3(ROOT_MIN),
         "colour": (C.c_float * 3)(1.0, 1.0, 1.0)}
    nv, nt = 1200000 * case["vpc"] // 64 + 65536, 800000 * case["vpc"] // 64 + 65536
    s["v"], s["t"] = _buffer((nv, 12), torch.float32, "device"), _buffer((nt, 3), torch.int32, "device")
    s["out"] = lvn.BatchOut(lvn.LVN_MEMORY_DEVICE, s["v"].data_ptr(), nv, 0, s["t"].data_ptr(), nt, 0, None, 0, 0,
                            C.cast(s["results"], C.POINTER(lvn.ChunkResult)))
    return s


def _prepare_collapse(case, seed):
    chunks, (V, T, _, res) = _meshes(case["vpc"], case["density"], seed)
    keep = np.flatnonzero(res[:, 3] > 0)[:case["meshes"]]
    v = np.concatenate([V[res[i, 0]:res[i, 0] + res[i, 1]] for i in keep])
    t = np.concatenate([T[res[i, 2]:res[i, 2] + res[i, 3]] for i in keep])
    ranges = np.zeros((len(keep), 8), np.int32)
    ranges[:, 1], ranges[:, 3] = res[keep, 1], res[keep, 3]
    ranges[1:, 0], ranges[1:, 2] = np.cumsum(ranges[:-1, 1]), np.cumsum(ranges[:-1, 3])
    s = {"m": len(keep), "ranges": ranges, "res": np.zeros_like(ranges),
         "offs": np.array([lvn.node_offset(*chunks[i]) for i in keep], np.float32),
         "opts": (lvn.SimplifyOptions * len(keep))(*[lvn.engine_simplify_options(chunks[i][1]) for i in keep]),
         "v": torch.from_numpy(v).cuda(), "t": torch.from_numpy(t).cuda()}
    s["ov"], s["ot"] = torch.empty_like(s["v"]), torch.empty_like(s["t"])
    # where the simplified meshes are packed for upload
    cap = 40000 * case["meshes"] * case["vpc"] ** 2 // 4096
    s["pv"], s["pt"] = _buffer((cap, 12), torch.float32, "device"), _buffer((2 * cap, 3), torch.int32, "device")
    return s


def _lattices(case, seed):
    rng = W.MT19937(seed + 71)
    span = case["step"] * (case["dim"] - 1)
    rows = []
    for _ in range(case["lattices"]):
        x, z = (math.floor(rng.uniform(-1024.0, 1024.0 - span)) for _ in range(2))
        rows.append([x, math.floor(rng.uniform(-128.0, 128.0 - span)), z, case["step"]])
    return np.array(rows, np.float32)


def _surrogate(case, seed):
    _world(case.get("density", "fbm2d"))
    sur = lvn.Surrogate(*DOMAIN, seed=seed % 9973 + 1)
    return sur


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("chunk", "edit"):
        _world(case["density"])
        mn, size = _surface_chunk(case["density"], case["vpc"], case["scale"], seed)
        cap = 9 * case["vpc"] ** 2 + 1024  # vertices and seam nodes; a chunk's surface has about 1.3 vpc^2
        s = {"mg": _context(case["vpc"], cache=1 if kind == "edit" else 0), "min": lvn._ivec3(mn), "size": size,
             "v": _buffer((cap, 12), torch.float32, "host"), "t": _buffer((2 * cap, 3), torch.int32, "host"),
             "s": _buffer((cap, 12), torch.int32, "host")}
        s["out"] = lvn.MeshOut(lvn.LVN_MEMORY_HOST, s["v"].data_ptr(), cap, 0, s["t"].data_ptr(), 2 * cap, 0,
                               s["s"].data_ptr(), cap, 0)
        if kind == "edit":
            m = s["mg"].generate_chunk_mesh(mn, size)  # the chunk as the player sees it
            centre = m.vertices[len(m.vertices) // 2, :3].astype(np.float64) / 4.0  # on its surface, density units
            r = case["radius"]
            s["ops"] = [[lvn.make_op(1, 1, W.MATERIAL_AIR, tuple(centre), (r, r, r))],
                        [lvn.make_op(0, 1, 1, tuple(centre), (r, r, r))]]
            s["turn"] = 0
    elif kind in ("tiles", "clipmap", "frame"):
        s = _prepare_batch(case, seed)
    elif kind == "select":
        _world("fbm2d")
        n = case["cameras"]
        cams = W.clipmap_cameras(-(-n // 64), 64, seed + 1)[:n]
        s = {"cams": cams, "memory": case["memory"]}
        if case["memory"] == "device":
            s["cams"] = torch.from_numpy(cams).cuda()
        s["nodes"] = _buffer((n * FRAME_MAX, 4), torch.int32, case["memory"])
        s["counts"] = _buffer((n,), torch.int32, case["memory"])
        s["rmin"] = lvn._ivec3(ROOT_MIN)
    elif kind == "seams":
        s = _prepare_seams(case, seed)
    elif kind == "collapse":
        s = _prepare_collapse(case, seed)
    elif kind == "train":
        s = {"sur": _surrogate(case, seed), "steps": case["steps"], "batch": case["batch"]}
        s["sur"].sample(1 << 20, seed=seed % 9973 + 1)
    else:
        lat = _lattices(case, seed)
        s = {"sur": _surrogate(case, seed), "lat": torch.from_numpy(lat).cuda(), "dim": case["dim"],
             "dens": torch.empty(len(lat) * case["dim"] ** 3, dtype=torch.float32, device="cuda")}
    s["kind"] = kind
    return s


# ---- run -----------------------------------------------------------------------


def _ok(rc, what):
    if rc < 0:
        raise lvn.LvnError(rc, what)


def run(s):
    kind = s["kind"]
    if kind in ("chunk", "edit"):
        if kind == "edit":  # dig, then fill, then dig again: each edit changes the field
            s["mg"].apply_csg_operations(s["ops"][s["turn"] & 1], s["min"], s["size"])
            s["turn"] += 1
            lvn.lib().lvn_meshgen_free_chunk_octree(s["mg"].handle, s["min"], s["size"])  # the mesh follows the field
        mo = s["out"]
        _ok(lvn.lib().lvn_meshgen_generate_chunk_mesh(s["mg"].handle, s["min"], s["size"], C.byref(mo)),
            "generate_chunk_mesh")
        return [s["v"], s["t"], s["s"], [mo.num_vertices, mo.num_triangles, mo.num_seams]]
    if kind in ("tiles", "clipmap", "frame"):
        bo = s["out"]
        _ok(s["mg"].generate_chunks_raw(s["descs"], s["n"], bo), "generate_chunks")
        return [s["v"], s["t"], s["s"], _rows(s["results"], s["rows"]),
                [bo.total_vertices, bo.total_triangles, bo.total_seams]]
    if kind == "select":
        if s["memory"] == "host":
            _ok(lvn.lib().lvn_clipmap_select(s["cams"].ctypes.data, len(s["cams"]), s["rmin"], ROOT_SIZE,
                                             s["nodes"].data_ptr(), len(s["nodes"]), s["counts"].data_ptr()),
                "clipmap_select")
        else:
            lvn.clipmap_select_device(s["cams"], ROOT_MIN, ROOT_SIZE, s["nodes"], FRAME_MAX, s["counts"])
        return [s["nodes"], s["counts"]]
    if kind == "seams":
        bo = s["out"]
        _ok(lvn.lib().lvn_seam_generate(s["descs"], s["offs"].ctypes.data, s["n"], s["rows"].data_ptr(),
                                        lvn.LVN_MEMORY_DEVICE, s["vpc"], s["rmin"], ROOT_SIZE, s["hosts"].ctypes.data,
                                        s["n"], s["colour"], C.byref(bo)), "seam_generate")
        return [s["v"], s["t"], _rows(s["results"], FRAME_MAX), [bo.total_vertices, bo.total_triangles]]
    if kind == "collapse":
        s["res"][:] = s["ranges"]
        _ok(lvn.lib().lvn_mesh_simplify(s["v"].data_ptr(), s["t"].data_ptr(), lvn.LVN_MEMORY_DEVICE,
                                        s["res"].ctypes.data_as(C.POINTER(lvn.ChunkResult)), s["m"],
                                        s["offs"].ctypes.data, s["opts"], s["ov"].data_ptr(), s["ot"].data_ptr()),
            "mesh_simplify")
        # only each range's first part holds its mesh now: pack them
        r = s["res"][:, :4].tolist()
        torch.cat([s["ov"][vo:vo + nv] for vo, nv, _, _ in r], out=s["pv"][:sum(x[1] for x in r)])
        torch.cat([s["ot"][to:to + nt] for _, _, to, nt in r], out=s["pt"][:sum(x[3] for x in r)])
        return [s["pv"], s["pt"], s["res"]]
    if kind == "train":
        losses = s["sur"].train(s["steps"], batch=s["batch"], lr=1e-3)
        return [losses, s["sur"].params()]
    _ok(lvn.lib().lvn_surrogate_eval_lattices(s["sur"]._h, s["lat"].data_ptr(), len(s["lat"]), s["dim"],
                                              s["dens"].data_ptr()), "surrogate_eval_lattices")
    return [s["dens"]]


# ---- what a pass cannot do without -------------------------------------------------

# FP32 operations of one density evaluation: the height term of each density
# (heightfield part) and the 3D term; counted as in tests/test_flop_counts.py
HEIGHT = {"terrain": 740.0, "fbm2d": 452.0, "caves": 452.0}
CAVE = {"terrain": 2.0, "fbm2d": 2.0, "caves": 601.0}


def _chunk_work(case, n, surface):
    """n chunks of which the share `surface` holds surface: a height per
    column, a sign per field point near the surface, a crossing and a normal
    (at least 2 + 6 densities) per edge and a vertex per leaf; the meshes
    written once."""
    v, d = case["vpc"], case["density"]
    leaves = surface * n * 1.3 * v * v
    edges = 1.5 * leaves
    flops = n * (v + 2) ** 2 * HEIGHT[d] + edges * (4 * HEIGHT[d] + 8 * CAVE[d] + 146.0) + leaves * 1500.0
    if d == "caves":
        flops += surface * n * (v + 2) ** 2 * 16 * CAVE[d]
    return {"bytes": leaves * (48 + 2 * 12) + surface * n * 4 * v * 48.0 + n * 64.0, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("chunk", "edit"):
        return _chunk_work(case, 1, 1.0)
    if kind == "tiles":
        return _chunk_work(case, case["nx"] * case["ny"] * case["nz"], min(1.0, 2.0 / case["ny"]))
    if kind == "clipmap":
        return _chunk_work(case, case["n"], 0.5)
    if kind == "frame":
        return _chunk_work(case, 420, 0.4)
    if kind == "select":
        return {"bytes": case["cameras"] * (12.0 + 410 * 16), "flops": case["cameras"] * 470 * 12.0}
    if kind == "seams":
        rows = 560.0 * 420 * case["vpc"] / 64
        return {"bytes": rows * 48 + 2.2 * rows * 48 + 1.35 * rows * 12, "flops": 2.2 * rows * 12 * 3 * 16.0}
    if kind == "collapse":
        v = case["meshes"] * 1.3 * case["vpc"] ** 2
        return {"bytes": v * (48 + 24) * 2, "flops": v * 3 * 0.125 * 10 * 2000.0}
    mlp = 2.0 * (96 * 128 + 3 * 128 * 128 + 128)
    if kind == "train":
        n = case["steps"] * case["batch"]
        return {"bytes": n * 16.0 + case["steps"] * 62081 * 4.0 * 6, "flops": 3 * mlp * n}
    n = case["lattices"] * case["dim"] ** 3
    return {"bytes": n * 4.0 + case["lattices"] * 16, "flops": mlp * n}


# ---- 64-bit values -------------------------------------------------------------


def exact(case, seed):
    """The surrogate's densities in 64 bits.  A mesh has no such value: which
    edges, leaves and triangles exist, and which of 17 samples is an edge's
    crossing, are decisions of the 32-bit density, and the rest of its numbers
    hang on them; the seams, selections and collapses copy or choose.  A
    training run's weights would take far too long."""
    if case["kind"] != "eval":
        return None
    state = prepare(case, seed)
    p = torch.from_numpy(state["sur"].params()).double().cuda()
    lat = torch.from_numpy(_lattices(case, seed)).double().cuda()
    dim, out = case["dim"], []
    widths, o, layers = [96, 128, 128, 128], 0, []
    for k in widths:
        layers.append((p[o:o + 128 * k].reshape(128, k), p[o + 128 * k:o + 128 * k + 128]))
        o += 128 * k + 128
    idx = torch.arange(dim, dtype=torch.float64, device="cuda")
    for x0, y0, z0, step in lat:
        z, y, x = torch.meshgrid(z0 + step * idx, y0 + step * idx, x0 + step * idx, indexing="ij")
        cols = []
        for a, c in enumerate((x, y, z)):
            ext = DOMAIN[1][a] - DOMAIN[0][a]
            freq = 2.0 ** (math.log2(max(2.0, ext / 2.0)) * torch.arange(16, dtype=torch.float64, device="cuda") / 15)
            ang = math.pi * (2.0 * (c.reshape(-1, 1) - DOMAIN[0][a]) / ext - 1.0) * freq
            cols += [torch.sin(ang), torch.cos(ang)]
        h = torch.cat(cols, 1)
        for w, b in layers:
            h = torch.nn.functional.silu(h @ w.T + b)
        out.append(8.0 * (h @ p[o:o + 128] + p[o + 128]))
    return [torch.cat(out)]

"""Workloads of the radiosity hot path, each through the entry points a caller uses.

Device buffers go through the ``_d`` functions of include/vradgpu.h, host arrays through the Python
face (``vrad_gb300.environment``).  Scenes are the seeded generators of ``vrad_gb300.scenes``: closed
box rooms, 4,096 units wide, with opaque boxes, a sky ceiling and point, spot and sky-ambient lights.
"""
import math

import numpy as np
import torch

from vrad_gb300 import scenes
from vrad_gb300.environment import Batch, Context, Environment, make_light

_CTX = None


def _ctx():
    """The process's one context, as a program that serves many scenes keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
    return _CTX


def listed():
    return [
        # One Trace4Rays call: the reference tracer's own granularity, the smallest call there is.
        {"name": "trace4", "kind": "trace4", "boxes": 1024},
        # TestLineDoesHitSky over a host array of lines, the size of a handful of leaves' sky sweeps.
        {"name": "sky_lines_host", "kind": "sky_lines", "faces": 1000, "n": 10007},
        # Closest hits of device-resident rays with ragged count, in a large map (49,164 triangles).
        {"name": "closest_rays", "kind": "closest", "boxes": 4096, "n": 262147},
        # The any-hit benchmark: 2^20 shadow lines against 12,300 triangles, device buffers.
        {"name": "mask_lines", "kind": "mask", "boxes": 1024, "n": 1 << 20},
        # Direct light of a small scene (the smallest of a batch), host arrays, 4 supersamples.
        {"name": "direct_small", "kind": "direct", "faces": 64, "spacing": 48.0, "tiles": 1, "brush": False, "ss": 4,
         "points": 64, "spots": 8, "host": True},
        # A preview bake of a compiled map's brushes: one sample per luxel, walls made of brush sides.
        {"name": "direct_brush_preview", "kind": "direct", "faces": 1001, "spacing": 16.0, "tiles": 1, "brush": True,
         "ss": 1, "points": 64, "spots": 8, "host": False},
        # The direct-light benchmark: 4,096 faces, 16-unit luxels, 4 supersamples, 72 lights and sky.
        {"name": "direct_full", "kind": "direct", "faces": 4096, "spacing": 16.0, "tiles": 1, "brush": False, "ss": 4,
         "points": 64, "spots": 8, "host": False},
        # Transfer lists of a small scene, read back to the host.
        {"name": "transfers_small", "kind": "transfers", "faces": 200, "k": 1024},
        # The radiosity benchmark: transfer lists at k = 65,536 for 4,096 faces, then the bounce loop.
        {"name": "radiosity_full", "kind": "radiosity", "faces": 4096, "k": 65536},
        # The bounce loop alone on resident transfer lists (a light table changed, the lists kept).
        {"name": "bounce", "kind": "bounce", "faces": 2731, "k": 8192},
        # Uneven scenes baked together, 48-unit luxels, and their results read back.
        {"name": "batch_bake", "kind": "bake", "scenes": 12, "lo": 64, "hi": 4096, "k": 8192},
        # A served light edit: two point lights moved, partial re-gather, warm bounce, results read back.
        {"name": "relight", "kind": "relight", "faces": 1000, "edits": 2, "k": 4096},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace4", "sky_lines", "closest", "mask", "direct", "direct", "transfers", "radiosity", "bounce",
                       "bake", "relight"])
    if kind == "trace4":
        return {"kind": kind, "boxes": _logint(rng, 64, 4096)}
    if kind == "sky_lines":
        return {"kind": kind, "faces": _logint(rng, 64, 4096), "n": _logint(rng, 33, 1 << 18)}
    if kind in ("closest", "mask"):
        return {"kind": kind, "boxes": _logint(rng, 64, 4096), "n": _logint(rng, 1 << 12, 1 << 20)}
    if kind == "direct":
        brush = rng.random() < 0.3
        faces = _logint(rng, 64, 4096)
        spacing = rng.choice([16.0, 24.0, 32.0, 48.0])
        return {"kind": kind, "faces": faces, "spacing": spacing,
                "tiles": 1 if brush else rng.choice([1, 1, 3, 16]), "brush": brush, "ss": rng.choice([1, 4]),
                "points": rng.randint(4, 64), "spots": rng.randint(0, 8), "host": faces <= 512}
    if kind == "transfers":
        return {"kind": kind, "faces": _logint(rng, 48, 400), "k": 1 << rng.randint(8, 12)}
    if kind in ("radiosity", "bounce"):
        return {"kind": kind, "faces": _logint(rng, 64, 4096 if kind == "radiosity" else 2731),
                "k": 1 << rng.randint(9, 16 if kind == "radiosity" else 13)}
    if kind == "bake":
        return {"kind": kind, "scenes": rng.randint(1, 12), "lo": 64, "hi": _logint(rng, 200, 4096),
                "k": 1 << rng.randint(10, 13)}
    return {"kind": kind, "faces": _logint(rng, 100, 2000), "edits": rng.randint(1, 8), "k": 1 << rng.randint(10, 12)}


# --- what a program has in hand before the call ------------------------------------------------


def _uniform(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _room(case, seed):
    sc = scenes.anyhit_scene(seed, n_boxes=case["boxes"], n_rays=1)
    env = Environment(_ctx())
    env.add_triangles(sc.xyz, sc.ids)
    env.SetupAccelerationStructure()
    return env, sc


def _lit_map(case, seed):
    """(lumps, lit): a lit room with the case's faces; lumps (a compiled map's arrays) for a brush map,
    else None and the triangles in ``lit``.  Corners lie on a quarter-unit grid, as editors place them."""
    faces, spacing, tiles = case["faces"], case.get("spacing", 16.0), case.get("tiles", 1)
    brush = case.get("brush", False)
    rs = np.random.RandomState(seed % (1 << 32))
    n = (faces + 5) // 6
    u = (0.5 + np.arange(1, n + 1)[:, None] * np.array([0.8191725, 0.6710436, 0.5497005])) % 1.0
    edge = np.floor(64.0 + 448.0 * u) + 0.5
    centre = np.round(4.0 * (edge / 2 + 1.0 + rs.rand(n, 3) * (scenes.ROOM - 2.0 - edge))) / 4.0
    mins, maxs = (centre - edge / 2).astype(np.float32), (centre + edge / 2).astype(np.float32)
    soup, tri_face, side = scenes.TriangleSoup(), [], float(scenes.ROOM)
    for k, (a, b, _, d) in enumerate(scenes.box_quads((0.0, 0.0, 0.0), (side, side, side))[0]):
        a, b, d = (np.asarray(x, np.float64) for x in (a, b, d))
        tid = scenes.TRACE_ID_SKY if k == 0 else scenes.TRACE_ID_OPAQUE
        for i in range(tiles):
            for j in range(tiles):
                at = [a + (b - a) * (p / tiles) + (d - a) * (q / tiles)
                      for p, q in ((i, j), (i + 1, j), (i + 1, j + 1), (i, j + 1))]
                soup.add_quad(tid, *(tuple(float(c) for c in p) for p in at))
    tri_face += [-1] * len(soup.ids)
    recs = []
    for i in range(n):
        quads, normals = scenes.box_quads(mins[i], maxs[i])
        for k, (q, nrm) in enumerate(zip(quads, normals)):
            soup.add_quad(scenes.TRACE_ID_OPAQUE, *q)
            f = 6 * i + k
            tri_face += [f, f] if f < faces else [-1, -1]
            if f < faces:
                ax = int(np.argmax(np.abs(nrm)))
                p, r = (ax + 1) % 3, (ax + 2) % 3
                lo, hi = np.min(q, axis=0), np.max(q, axis=0)
                eu, ev = np.zeros(3), np.zeros(3)
                eu[p], ev[r] = hi[p] - lo[p], hi[r] - lo[r]
                recs.append((lo, eu, ev, nrm, math.ceil(eu[p] / spacing), math.ceil(ev[r] / spacing)))
    corner, eu, ev, nrm, nu, nv = (np.array([r[c] for r in recs]) for c in range(6))
    lights = []
    for i in range(case.get("points", 64) + case.get("spots", 8)):
        spot = i >= case.get("points", 64)
        keys = dict(quadratic_attn=1.0, distance=1024.0)
        if spot:
            keys.update(inner_cone=30.0, cone=45.0, exponent=1.0)
        aim = rs.randn(3)
        aim = tuple(float(c) for c in (aim / np.linalg.norm(aim)).astype(np.float32)) if spot else (0.0, 0.0, -1.0)
        lights.append(scenes.Light(scenes.EMIT_SPOTLIGHT if spot else scenes.EMIT_POINT,
                                   tuple(float(c) for c in rs.uniform(1.0, side - 1.0, 3).astype(np.float32)),
                                   tuple(float(c) for c in rs.uniform(50.0, 500.0, 3).astype(np.float32)), aim, keys))
    lights.append(scenes.Light(scenes.EMIT_SKYAMBIENT, (0.0, 0.0, 0.0), (40.0, 50.0, 70.0)))
    f32 = lambda x: np.ascontiguousarray(x, np.float32)  # noqa: E731
    xyz, ids = soup.arrays()
    lit = scenes.LitScene(xyz, ids, np.asarray(tri_face, np.int32), f32(corner), f32(eu), f32(ev), f32(nrm),
                          nu.astype(np.int32), nv.astype(np.int32), np.full(faces, 1.0 / spacing, np.float32),
                          f32(rs.uniform(0.1, 0.8, (faces, 3))), lights)
    if not brush:
        return None, lit
    # the same room as a compiled map's brushes: floor and walls 16 units thick, a sky face, one brush a box
    w, t = scenes.BrushMap(), 16.0
    w.box((-t, -t, -t), (side + t, side + t, 0.0))
    w.box((-t, -t, 0.0), (0.0, side + t, side))
    w.box((side, -t, 0.0), (side + t, side + t, side))
    w.box((0.0, -t, 0.0), (side, 0.0, side))
    w.box((0.0, side, 0.0), (side, side + t, side))
    w.face([(0.0, 0.0, side), (side, 0.0, side), (side, side, side), (0.0, side, side)], texinfo=1)
    tri_face = [-1] * 60
    for i in range(n):
        w.box(tuple(float(c) for c in mins[i]), tuple(float(c) for c in maxs[i]))
        for k in (3, 2, 4, 5, 0, 1):  # brush sides +x -x +y -y +z -z as faces of box_quads
            f = 6 * i + k
            tri_face += [f, f] if f < faces else [-1, -1]
    lit.tri_face = np.asarray(tri_face + [-1, -1], np.int32)
    return w.lumps(), lit


def _lit_env(lit, lumps=None):
    env = Environment(_ctx())
    if lumps is not None:
        env.add_bsp_world(lumps)
    else:
        env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    return env


def _segments(seed, n):
    p = 1.0 + (scenes.ROOM - 2.0) * _uniform(seed, 2, n, 3)
    return p[0].contiguous(), p[1].contiguous()


def _rays(seed, n):
    """Origins in the room and unit directions towards a second point, range [0, MAX_TRACE_LENGTH)."""
    a, b = _segments(seed, n)
    d = torch.nn.functional.normalize(b - a, dim=1)
    return a, d, torch.zeros(n, device="cuda"), torch.full((n,), 56755.84, device="cuda")


def _edits(lit, seed, n):
    """Two edit lists: `n` point lights moved elsewhere, and moved back."""
    rs = np.random.RandomState(seed % (1 << 31))
    idx = rs.permutation(np.flatnonzero([li.type == scenes.EMIT_POINT for li in lit.lights]))[:n]
    out, back = [], []
    for i in idx:
        li = lit.lights[i]
        moved = scenes.Light(li.type, tuple(float(c) for c in rs.uniform(64.0, scenes.ROOM - 64.0, 3)), li.intensity,
                             li.normal, li.keys)
        out.append((int(i), make_light(moved.type, moved.origin, moved.intensity, moved.normal, **moved.keys)))
        back.append((int(i), make_light(li.type, li.origin, li.intensity, li.normal, **li.keys)))
    return [out, back]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("trace4", "closest", "mask"):
        st["env"], st["scene"] = _room(case, seed)
        if kind == "trace4":
            o, d, t0, t1 = (x.cpu().numpy() for x in _rays(seed, 4))
            st["rays"] = (np.ascontiguousarray(o.T).ravel(), np.ascontiguousarray(d.T).ravel(), t0, t1)
        elif kind == "closest":
            st["rays"] = _rays(seed, case["n"])
            st["hit"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
            st["t"] = torch.empty(case["n"], dtype=torch.float32, device="cuda")
        else:
            st["lines"] = _segments(seed, case["n"])
            st["mask"] = torch.empty((case["n"] + 31) // 32, dtype=torch.int32, device="cuda")
    elif kind == "sky_lines":
        _, lit = _lit_map(case, seed)
        st["env"], st["scene"] = _lit_env(lit), lit
        st["lines"] = tuple(x.cpu().numpy() for x in _segments(seed, case["n"]))
    elif kind == "direct":
        lumps, lit = _lit_map(case, seed)
        st["env"], st["scene"] = _lit_env(lit, lumps), lit
        if not case["host"]:
            st["rgb"] = torch.empty(st["env"].num_luxels(), 3, dtype=torch.float32, device="cuda")
    elif kind == "bake":
        n = case["scenes"]
        counts = [case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / n) for i in range(n)]
        dirs = scenes.transfer_directions(case["k"])
        st["envs"], st["leaves"] = [], []
        for i, f in enumerate(counts):
            env = _lit_env(_lit_map({"faces": int(f), "spacing": 48.0}, 1000 * seed + i)[1])
            st["leaves"].append(env.make_patches()["n_leaves"])
            env.make_transfers(dirs)
            st["envs"].append(env)
        if len(counts) > 1:
            st["batch"] = Batch(_ctx())
            for env in st["envs"]:
                st["batch"].add(env)
    else:  # transfers, radiosity, bounce, relight
        _, lit = _lit_map(dict(case, spacing=48.0) if kind == "relight" else case, seed)
        env = _lit_env(lit)
        patches = env.make_patches()
        st["env"], st["scene"], st["leaves"] = env, lit, patches["n_leaves"]
        st["dirs"] = scenes.transfer_directions(case["k"])
        if kind in ("radiosity", "bounce"):
            st["direct"] = env.gather_patch_direct(st["leaves"])
        if kind in ("bounce", "relight"):
            st["nnz"] = env.make_transfers(st["dirs"])
        if kind == "transfers":  # the caller's arrays; a row has at most k entries, in these maps under k / 4
            cap = st["leaves"] * case["k"] // 4
            st["csr"] = (np.zeros(st["leaves"] + 1, np.int64), np.zeros(cap, np.int32), np.zeros(cap, np.float32))
        if kind == "bounce":
            leaf = patches["leaf_index"] >= 0
            face = np.empty(st["leaves"], np.int64)
            face[patches["leaf_index"][leaf]] = patches["face"][leaf]
            st["refl"] = lit.refl[face]
        if kind == "relight":
            env.relight_prepare()
            st["edits"], st["turn"] = _edits(lit, seed, case["edits"]), 0
    torch.cuda.synchronize()
    return st


# --- one pass ----------------------------------------------------------------------------------


def _ok(env, rc):
    if rc != 0:
        raise RuntimeError(env.lib.vrg_last_error(env.ctx.h).decode())


def _run_trace4(st):
    o, d, t0, t1 = st["rays"]
    return st["env"].Trace4Rays(o, d, t0, t1)


def _run_sky_lines(st):
    return st["env"].test_line_does_hit_sky(*st["lines"])


def _run_closest(st):
    env = st["env"]
    o, d, t0, t1 = st["rays"]
    _ok(env, env.lib.vrg_env_trace_closest_d(env.h, o.data_ptr(), d.data_ptr(), t0.data_ptr(), t1.data_ptr(),
                                             o.shape[0], -1, st["hit"].data_ptr(), st["t"].data_ptr()))
    return st["hit"], st["t"]


def _run_mask(st):
    env = st["env"]
    a, b = st["lines"]
    _ok(env, env.lib.vrg_env_occlusion_mask_d(env.h, a.data_ptr(), b.data_ptr(), a.shape[0], -1,
                                              st["mask"].data_ptr(), None, None))
    return st["mask"]


def _run_direct(st):
    env, case = st["env"], st["case"]
    if case["host"]:
        return env.gather_direct_light(case["ss"], 0)
    _ok(env, env.lib.vrg_env_gather_direct_light_d(env.h, case["ss"], 0, st["rgb"].data_ptr(), None))
    return st["rgb"]


def _run_transfers(st):
    env = st["env"]
    row, col, w = st["csr"]
    if env.make_transfers(st["dirs"]) > col.size:
        raise RuntimeError("more transfers than the arrays hold")
    _ok(env, env.lib.vrg_env_get_transfers(env.h, row.ctypes.data, col.ctypes.data, w.ctypes.data))
    return st["csr"]


def _run_radiosity(st):
    nnz = st["env"].make_transfers(st["dirs"])
    total, bounces, _ = st["env"].bounce_light(st["leaves"])
    return {"nnz": nnz, "total": total, "bounces": bounces}


def _run_bounce(st):
    total, bounces, _ = st["env"].bounce_light(st["leaves"])
    return {"total": total, "bounces": bounces}


def _run_bake(st):
    if len(st["envs"]) > 1:
        st["batch"].bake()
    else:
        st["envs"][0].bake()
    out = []
    for env, n in zip(st["envs"], st["leaves"]):
        b = env.get_bake(n)
        out.append([b["luxels"], b["patch_direct"], b["patch_total"], b["bounces"]])
    return out


def _run_relight(st):
    edits = st["edits"][st["turn"]]
    st["turn"] ^= 1
    st["env"].relight(edits)
    b = st["env"].get_bake(st["leaves"])
    return {k: b[k] for k in ("luxels", "patch_direct", "patch_total")}


_RUN = {"trace4": _run_trace4, "sky_lines": _run_sky_lines, "closest": _run_closest, "mask": _run_mask,
        "direct": _run_direct, "transfers": _run_transfers, "radiosity": _run_radiosity, "bounce": _run_bounce,
        "bake": _run_bake, "relight": _run_relight}


def run(state):
    return _RUN[state["kind"]](state)


# --- what a pass cannot do without ---------------------------------------------------------------

_TEST = 45  # operations of one ray/triangle test


def _luxels(faces, spacing):
    """Expected luxels: box edges are uniform in [64, 512]."""
    return faces * (288.0 / spacing + 0.5) ** 2


def work(case):
    kind = case["kind"]
    tri = 48.0 * (12 + 12 * case.get("boxes", (case.get("faces", 64) + 5) // 6))
    if kind == "trace4":
        return {"bytes": 4 * 32 + 4 * 20 + 4 * 48, "flops": 4 * _TEST}
    if kind == "sky_lines":
        return {"bytes": 28 * case["n"] + tri, "flops": case["n"] * _TEST}
    if kind == "closest":
        return {"bytes": 40 * case["n"] + tri, "flops": case["n"] * _TEST}
    if kind == "mask":
        return {"bytes": 24.125 * case["n"] + tri, "flops": case["n"] * _TEST}
    if kind == "direct":  # half the 162 sky directions of each sample, one test each; 12 bytes a luxel
        lux = _luxels(case["faces"], case["spacing"])
        return {"bytes": 12 * lux + tri, "flops": lux * case["ss"] * 81 * _TEST}
    if kind == "bake":  # log-uniform face counts, 35 leaf patches a face, about 8 bounces over the lists
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        lux, leaves = _luxels(mean, 48.0) * case["scenes"], 35.0 * mean * case["scenes"]
        nnz = leaves * min(case["k"] / 16.0, 500.0)
        return {"bytes": 12 * lux + 24 * leaves + 8 * nnz, "flops": (4 * lux + leaves) * 81 * _TEST + 48 * nnz}
    leaves = 35.0 * case["faces"]
    if kind == "relight":  # the sky is cached: what moves is the light edits' faces and the warm bounces
        nnz = leaves * case["k"] / 16.0
        return {"bytes": 12 * _luxels(case["faces"], 48.0) + 24 * leaves + 8 * nnz, "flops": 4 * 6 * nnz}
    rays = leaves * case["k"]
    nnz = leaves * min(case["k"] / 16.0 if case["k"] <= 16384 else case["k"] / 34.0, leaves)
    if kind == "transfers":
        return {"bytes": 8 * nnz + tri, "flops": rays * _TEST}
    if kind == "radiosity":
        return {"bytes": 16 * nnz + tri, "flops": rays * _TEST + 8 * 6 * nnz}
    return {"bytes": 8 * nnz + 64 * leaves, "flops": 8 * 6 * nnz}


# --- the same in 64 bits -------------------------------------------------------------------------


def _closest64(xyz, o, d, tmax):
    """(t, index) of the closest hit on [0, tmax) by testing every triangle in float64; t = inf, -1 for none."""
    v = torch.as_tensor(np.asarray(xyz), device="cuda").double().view(-1, 3, 3)
    n = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    nn = (n * n).sum(1)
    dist = (n * v[:, 0]).sum(1)
    # barycentric rows: b_k = e_k . h + c_k
    e1 = torch.linalg.cross(n, v[:, 0] - v[:, 2]) / nn[:, None]
    c1 = -(e1 * v[:, 2]).sum(1)
    e2 = torch.linalg.cross(n, v[:, 1] - v[:, 0]) / nn[:, None]
    c2 = -(e2 * v[:, 0]).sum(1)
    o, d, tmax = o.double(), d.double(), tmax.double()
    ts, ids = [], []
    step = max(1, (1 << 27) // max(1, v.shape[0]))
    for i in range(0, o.shape[0], step):
        oo, dd = o[i:i + step], d[i:i + step]
        t = (dist - oo @ n.T) / (dd @ n.T)
        b1 = oo @ e1.T + t * (dd @ e1.T) + c1
        b2 = oo @ e2.T + t * (dd @ e2.T) + c2
        hit = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= 0) & (t < tmax[i:i + step, None])
        t = torch.where(hit, t, torch.full_like(t, math.inf))
        m, k = t.min(dim=1)
        ts.append(m)
        ids.append(torch.where(torch.isinf(m), torch.full_like(k, -1), k))
    return torch.cat(ts), torch.cat(ids)


def _visible64(lit, a, b):
    """1.0 where the segment a -> b is stopped by nothing, or by a sky triangle first."""
    d = b.double() - a.double()
    length = d.norm(dim=1)
    _, k = _closest64(lit.xyz, a, d / length[:, None], length)
    ids = torch.as_tensor(lit.ids, device="cuda")
    return ((k < 0) | ((ids[k.clamp(min=0)] & scenes.TRACE_ID_SKY) != 0)).double()


def _sky_directions():
    """The 162 sky directions: an icosahedron's faces cut into 16, pushed out to the sphere, six decimals."""
    x, z = 0.525731112119133606, 0.850650808352039932
    ico = np.array([(-x, 0, z), (x, 0, z), (-x, 0, -z), (x, 0, -z), (0, z, x), (0, z, -x), (0, -z, x), (0, -z, -x),
                    (z, x, 0), (-z, x, 0), (z, -x, 0), (-z, -x, 0)])
    near = np.abs(np.linalg.norm(ico[:, None] - ico[None], axis=2) - 2 * x) < 1e-9
    found = set()
    for i in range(12):
        for j in range(i):
            for k in range(j):
                if near[i, j] and near[i, k] and near[j, k]:
                    for p in range(5):
                        for q in range(5 - p):
                            s = (p * ico[i] + q * ico[j] + (4 - p - q) * ico[k]) / 4
                            found.add(tuple(np.round(s / np.linalg.norm(s), 6) + 0.0))
    return torch.tensor(sorted(found), dtype=torch.float64, device="cuda")


def _mix(i):
    """SplitMix64 of seed 0 at counter i."""
    with np.errstate(over="ignore"):
        z = (i.astype(np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _samples64(lit, ss):
    """Sample points and normals, luxel by luxel, ss of them each."""
    pts, nrm, first = [], [], 0
    for f in range(lit.n_faces):
        nu, nv = int(lit.nu[f]), int(lit.nv[f])
        lux = np.repeat(np.arange(nu * nv, dtype=np.int64), ss)
        k = np.tile(np.arange(ss), nu * nv)
        iu, iv = lux % nu, lux // nu
        if ss == 4:
            h = _mix((first + lux) * 4 + k)
            r1 = (h >> np.uint64(40)).astype(np.float64) * 2.0 ** -24
            r2 = ((h >> np.uint64(16)) & np.uint64(0xFFFFFF)).astype(np.float64) * 2.0 ** -24
            su, sv = (iu + ((k & 1) + r1) * 0.5) / nu, (iv + ((k >> 1) + r2) * 0.5) / nv
        else:
            su, sv = (iu + 0.5) / nu, (iv + 0.5) / nv
        n = lit.normal[f].astype(np.float64)
        pts.append(lit.corner[f].astype(np.float64) + su[:, None] * lit.u[f].astype(np.float64)
                   + sv[:, None] * lit.v[f].astype(np.float64) + 0.125 * n)
        nrm.append(np.broadcast_to(n, (lux.size, 3)))
        first += nu * nv
    return (torch.as_tensor(np.concatenate(x), device="cuda") for x in (pts, nrm))


def _direct64(lit, ss):
    """Direct light of every luxel: point and spot lights with 1/d^2 falloff inside their radius, the sky by
    the cosine-weighted share of the 162 directions that reach it."""
    p, n = _samples64(lit, ss)
    out = torch.zeros_like(p)
    lines = 0
    for li in lit.lights:
        rgb = torch.tensor(np.asarray(li.intensity, np.float32).astype(np.float64), device="cuda")
        if li.type == scenes.EMIT_SKYAMBIENT:
            total, seen = torch.zeros(len(p), device="cuda").double(), torch.zeros(len(p), device="cuda").double()
            for a in _sky_directions():
                w = n @ a
                at = torch.nonzero(w > 0).ravel()
                total[at] += w[at]
                seen[at] += w[at] * _visible64(lit, p[at], p[at] + a * 56755.84)
                lines += len(at)
            out += torch.where(total > 0, seen / total, torch.zeros_like(total))[:, None] * rgb
            continue
        o = torch.tensor(np.asarray(li.origin, np.float32).astype(np.float64), device="cuda")
        d = o - p
        r = d.norm(dim=1)
        d = d / r[:, None]
        cos = (n * d).sum(1)
        f = 1.0e4 / (r * r)
        lit_by = (cos > 0) & (r <= li.keys["distance"])
        if li.type == scenes.EMIT_SPOTLIGHT:
            c = -(d @ torch.tensor(np.asarray(li.normal, np.float32).astype(np.float64), device="cuda"))
            inner, outer = math.cos(math.radians(li.keys["inner_cone"])), math.cos(math.radians(li.keys["cone"]))
            lit_by &= c > outer
            f = f * c * ((c - outer) / (inner - outer)).clamp(max=1.0)
        at = torch.nonzero(lit_by).ravel()
        lines += len(at)
        if len(at):
            out[at] += (f[at] * cos[at] * _visible64(lit, p[at], o.expand(len(at), 3)))[:, None] * rgb
    return out.view(-1, ss, 3).mean(dim=1), lines


def exact(case, seed):
    kind = case["kind"]
    if kind in ("trace4", "closest"):
        sc = scenes.anyhit_scene(seed, n_boxes=case["boxes"], n_rays=1)
        o, d, _, t1 = _rays(seed, 4 if kind == "trace4" else case["n"])
        if kind == "closest" and case["n"] * (12.0 + 12 * case["boxes"]) > 2e10:
            return None
        t, k = _closest64(sc.xyz, o, d, t1)
        if kind == "closest":
            return None, t
        v = torch.as_tensor(sc.xyz, device="cuda").double().view(-1, 3, 3)[k]
        nrm = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        return None, t, nrm.T.reshape(-1)
    if kind == "sky_lines":
        a, b = _segments(seed, case["n"])
        return _visible64(_lit_map(case, seed)[1], a, b)
    if kind == "direct":
        # a brush map's triangles come out of the library, and the larger scenes take minutes
        lux = _luxels(case["faces"], case["spacing"]) * case["ss"]
        if case["brush"] or lux * 100 * (12 * case["tiles"] ** 2 + 2 * case["faces"]) > 5e9:
            return None
        rgb, lines = _direct64(_lit_map(case, seed)[1], case["ss"])
        return (rgb, lines) if case["host"] else rgb
    if kind == "bounce":
        # the lists are this case's input; the loop in float64 over them
        st = prepare(case, seed)
        row, col, w = st["env"].get_transfers(st["leaves"], st["nnz"])
        m = torch.sparse_csr_tensor(torch.as_tensor(row), torch.as_tensor(col.astype(np.int64)),
                                    torch.as_tensor(w).double(), (st["leaves"],) * 2).cuda()
        refl, direct = (torch.as_tensor(x, device="cuda").double() for x in (st["refl"], st["direct"]))
        emit, total, bounces = refl * direct, torch.zeros_like(direct), 0
        while bounces < 100:
            add = m @ emit
            total += add
            emit = refl * add
            bounces += 1
            if float(add.abs().sum() / total.abs().sum()) < 1e-3:
                break
        return {"total": total, "bounces": bounces}
    # transfer weights are ray counts over k, equal or a different list; the whole bakes' rays are too many
    return None

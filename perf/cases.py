"""Timed workloads of the framework, each through its public entry points.

A case is one call (or one short sequence of calls) that a user's program
makes again and again: a BLAS build, a scene build, a per-frame TLAS rebuild,
a trace, a training step of the split proposer. ``listed()`` names the ones
that are quoted; ``draw(rng)`` gives others of the same ranges. Inputs are
made on the GPU from the seed alone.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from marigold_b200 import _lib, learned, synth
from marigold_b200.bvh import (BoundingVolumeHierarchy, BvhSettings, Scene, build_batch_device, build_device,
                               default_context, instance_aabbs_device, trace_scene_device)


def listed():
    return [
        # A render loop's TLAS over a few hundred instances, rebuilt every
        # frame without an allocation: launches and latency are all of it.
        {"name": "tlas_noalloc_777", "kind": "tlas_noalloc", "n": 777},
        # The same frame step for a full scene: the instances' world boxes
        # from their transforms, then the TLAS over them.
        {"name": "tlas_frame_4096", "kind": "tlas_frame", "n": 4096, "meshes": 512},
        # One mesh of a model file, in the 16-bin profile with the adaptive
        # sweep off.
        {"name": "blas_random_65536_bins16", "kind": "blas", "mesh": "random", "n": 65536, "profile": "bins16",
         "min_leaf": 1, "max_leaf": 1},
        # The headline build: the noisy level-8 icosphere, one object per leaf.
        {"name": "blas_icosphere_l8", "kind": "blas", "mesh": "icosphere", "n": 1310720, "profile": "reference",
         "min_leaf": 1, "max_leaf": 1},
        # A ragged mesh with leaves of up to four objects (the compaction path).
        {"name": "blas_icosphere_300007_leaf4", "kind": "blas", "mesh": "icosphere", "n": 300007,
         "profile": "reference", "min_leaf": 1, "max_leaf": 4},
        # The largest single build: blobs, a ground grid and thin triangles.
        {"name": "blas_mixed_16m", "kind": "blas", "mesh": "mixed", "n": 16777216, "profile": "reference",
         "min_leaf": 1, "max_leaf": 1},
        # A whole scene at load time: 512 meshes and the TLAS in one call,
        # rebuilt with its captured graph.
        {"name": "batch_512_meshes", "kind": "batch", "meshes": 512, "largest": 262144, "instances": 4096},
        # The crate's own call on host lists, copies and permutation included.
        {"name": "host_new_327680", "kind": "host", "n": 327680},
        # The learned form at its recommended gate.
        {"name": "learned_icosphere_l8", "kind": "learned", "mesh": "icosphere", "n": 1310720},
        # Closest hits of random rays in a large scene, one BLAS.
        {"name": "trace_mixed_2m_rays", "kind": "trace", "n": 4194304, "rays": 2097152, "wide": False},
        # Closest hits through the two-level scene.
        {"name": "trace_scene_4m_rays", "kind": "trace_scene", "meshes": 512, "largest": 65536, "instances": 4096,
         "rays": 4194304},
        # One training step of the split proposer: gradients, then Adam.
        {"name": "train_4096", "kind": "train", "batch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tlas_noalloc", "tlas_frame", "blas", "blas", "blas", "batch", "host", "learned", "trace",
                       "trace", "trace_scene", "train"])
    if kind == "tlas_noalloc":
        return {"kind": kind, "n": _log_int(rng, 40, 1024)}
    if kind == "tlas_frame":
        return {"kind": kind, "n": _log_int(rng, 1025, 32768), "meshes": rng.randint(16, 512)}
    if kind == "blas":
        mesh = rng.choice(["random", "icosphere", "mixed"])
        top = {"random": 2097152, "icosphere": 1310720, "mixed": 8388608}[mesh]
        leaf = rng.choice([(1, 1), (1, 1), (1, 2), (1, 4), (2, 4)])
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 5000, top),
                "profile": rng.choice(["reference", "reference", "bins16", "steps16"]),
                "min_leaf": leaf[0], "max_leaf": leaf[1]}
    if kind == "batch":
        return {"kind": kind, "meshes": rng.randint(64, 512), "largest": _log_int(rng, 8192, 131072),
                "instances": _log_int(rng, 256, 4096)}
    if kind == "host":
        return {"kind": kind, "n": _log_int(rng, 20000, 1310720)}
    if kind == "learned":
        return {"kind": kind, "mesh": rng.choice(["random", "icosphere"]), "n": _log_int(rng, 65536, 1310720)}
    if kind == "trace":
        return {"kind": kind, "n": _log_int(rng, 65536, 4194304), "rays": _log_int(rng, 65536, 2097152),
                "wide": rng.random() < 0.5}
    if kind == "trace_scene":
        return {"kind": kind, "meshes": rng.randint(64, 512), "largest": _log_int(rng, 4096, 65536),
                "instances": _log_int(rng, 256, 4096), "rays": _log_int(rng, 65536, 4194304)}
    return {"kind": kind, "batch": _log_int(rng, 256, 16384)}


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _unit(shape, g):
    v = torch.randn(*shape, 3, device="cuda", generator=g)
    return v / v.norm(dim=-1, keepdim=True).clamp_min(1e-20)


def _uniform(shape, lo, hi, g):
    return lo + (hi - lo) * torch.rand(*shape, device="cuda", generator=g)


@functools.lru_cache(maxsize=None)
def _icosphere(level):
    """The unit icosphere's vertices and faces (no seed in them)."""
    v, f = synth.icosphere(level)
    return torch.from_numpy(v).cuda(), torch.from_numpy(f.astype(np.int32)).cuda()


def _value_noise(p, g):
    """Three octaves of value noise on a random lattice, in [-1, 1]."""
    total = torch.zeros(p.shape[0], device="cuda", dtype=torch.float64)
    for freq, amp in ((1.0, 1.0), (2.0, 0.5), (4.0, 0.25)):
        lattice = _uniform((12, 12, 12), -1.0, 1.0, g).double()
        q = p * freq
        i = q.floor()
        t = q - i
        w = t * t * (3.0 - 2.0 * t)
        i = i.long() + 6
        for c in range(8):
            d = [(c >> k) & 1 for k in range(3)]
            weight = torch.ones_like(total)
            for k in range(3):
                weight = weight * (w[:, k] if d[k] else 1.0 - w[:, k])
            total += amp * weight * lattice[i[:, 0] + d[0], i[:, 1] + d[1], i[:, 2] + d[2]]
    return total / 1.75


def _mesh_vertices(pos):
    """MeshVertex records (32 bytes, position first)."""
    v = torch.zeros(pos.shape[0], 8, device="cuda", dtype=torch.float32)
    v[:, :3] = pos.float() + 0.0
    return v


def _unshared(corners):
    """[N, 3, 3] corners as unshared vertices and index triples."""
    n = corners.shape[0]
    return corners.reshape(3 * n, 3), torch.arange(3 * n, device="cuda", dtype=torch.int32).reshape(n, 3)


def _random_mesh(n, g):
    v0 = torch.rand(n, 3, device="cuda", generator=g)
    e = _unit((n, 2), g) * _uniform((n, 2, 1), 0.001, 0.02, g)
    pos, tris = _unshared(torch.stack([v0, v0 + e[:, 0], v0 + e[:, 1]], 1))
    return _mesh_vertices(pos), tris


def _icosphere_mesh(n, g):
    level = 0
    while 20 * 4 ** level < n:
        level += 1
    p, f = _icosphere(level)
    return _mesh_vertices(p * (1.0 + 0.05 * _value_noise(p, g))[:, None]), f[:n].contiguous()


def _mixed_mesh(n, g):
    """Half the triangles small ones in 64 Gaussian blobs, a quarter a flat
    ground grid, the rest long thin ones; unshared 12-byte vertices."""
    nb = n // 2
    gx = max(2, int(math.sqrt(n / 4)))
    gz = max(1, (n // 4) // (2 * gx))
    nt = n - nb - 2 * gx * gz
    centre = torch.stack([_uniform((64,), -80.0, 80.0, g), _uniform((64,), 0.0, 60.0, g),
                          _uniform((64,), -80.0, 80.0, g)], -1)
    sigma = _uniform((64,), 0.5, 5.0, g)
    which = torch.arange(nb, device="cuda") % 64
    v0 = centre[which] + sigma[which, None] * torch.randn(nb, 3, device="cuda", generator=g)
    e = _unit((nb, 2), g) * _uniform((nb, 2, 1), 0.02, 0.2, g)
    blobs = torch.stack([v0, v0 + e[:, 0], v0 + e[:, 1]], 1)
    xs = torch.linspace(-100.0, 100.0, gx + 1, device="cuda")
    zs = torch.linspace(-100.0, 100.0, gz + 1, device="cuda")
    qx, qz = torch.meshgrid(torch.arange(gx, device="cuda"), torch.arange(gz, device="cuda"), indexing="ij")
    qx, qz = qx.reshape(-1), qz.reshape(-1)

    def corner(dx, dz):
        return torch.stack([xs[qx + dx], torch.zeros_like(xs[qx]), zs[qz + dz]], -1)

    ground = torch.stack([torch.stack([corner(0, 0), corner(1, 0), corner(1, 1)], 1),
                          torch.stack([corner(0, 0), corner(1, 1), corner(0, 1)], 1)], 1).reshape(-1, 3, 3)
    c = torch.stack([_uniform((nt,), -100.0, 100.0, g), _uniform((nt,), 0.0, 60.0, g),
                     _uniform((nt,), -100.0, 100.0, g)], -1)
    length = _uniform((nt, 1), 2.0, 10.0, g)
    u = _unit((nt,), g)
    w = torch.linalg.cross(u, _unit((nt,), g))
    w = w / w.norm(dim=-1, keepdim=True).clamp_min(1e-20)
    thin = torch.stack([c - 0.5 * length * u, c + 0.5 * length * u, c + length / 200.0 * w], 1)
    pos, tris = _unshared(torch.cat([blobs, ground, thin]))
    return pos.float().contiguous() + 0.0, tris


def _mesh(kind, n, g):
    return {"random": _random_mesh, "icosphere": _icosphere_mesh, "mixed": _mixed_mesh}[kind](n, g)


def _bounds(v):
    """A mesh's accessor bounds, as its file gives them."""
    return torch.cat([v[:, :3].amin(0), v[:, :3].amax(0)]).cpu().numpy()


def _transforms(n, g):
    """Column-major instance transforms: rotation, uniform scale in [0.5, 2],
    translation in [-100, 100]^3."""
    q = torch.randn(n, 4, device="cuda", generator=g)
    x, y, z, w = (q / q.norm(dim=1, keepdim=True).clamp_min(1e-20)).unbind(1)
    rot = torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
        torch.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
        torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], 1)
    m = torch.zeros(n, 4, 4, device="cuda")
    m[:, :3, :3] = rot.transpose(1, 2) * _uniform((n, 1, 1), 0.5, 2.0, g)
    m[:, 3, :3] = _uniform((n, 3), -100.0, 100.0, g)
    m[:, 3, 3] = 1.0
    return m.reshape(n, 16).contiguous() + 0.0


def _instances(n, bounds, g):
    """(mesh of each instance, transforms) over the meshes of `bounds`."""
    ids = torch.randint(0, bounds.shape[0], (n,), device="cuda", generator=g, dtype=torch.int32)
    return ids, _transforms(n, g)


def _rays(n, lo, hi, g):
    """Origins uniform in the box grown by a tenth, directions uniform."""
    ext = hi - lo
    r = torch.zeros(n, 8, device="cuda")
    r[:, :3] = lo - 0.1 * ext + 1.2 * ext * torch.rand(n, 3, device="cuda", generator=g)
    r[:, 4:7] = _unit((n,), g)
    return r


def _settings(case, bounds=None):
    s = BvhSettings(bounds=bounds)
    profile = case.get("profile", "reference")
    if profile == "bins16":
        s.bins, s.adaptive_max_n = 16, 0
    elif profile == "steps16":
        s.bins, s.adaptive_steps = 32, 16
    return s


def _outputs(n):
    slots = max(2 * n - 1, 1)
    return {"nodes": torch.zeros(slots * 8, dtype=torch.int32, device="cuda"),
            "lens": torch.zeros(slots, dtype=torch.int32, device="cuda"),
            "perm": torch.zeros(n, dtype=torch.int32, device="cuda")}


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


def _scene(case, g):
    """Meshes of log-uniform sizes (random or icosphere, by a coin) and their
    instances, as one batched build's descriptors. The sizes are spread by the
    golden ratio, so a case's total does not vary with the seed."""
    m = case["meshes"]
    coin = torch.rand(m, device="cuda", generator=g).cpu().numpy()
    spread = (np.arange(1, m + 1) * 0.6180339887498949) % 1.0
    sizes = np.rint(64.0 * (case["largest"] / 64.0) ** spread).astype(np.int64)
    meshes = [_mesh("random" if coin[k] < 0.5 else "icosphere", int(sizes[k]), g) for k in range(m)]
    boxes = torch.stack([torch.cat([v[:, :3].amin(0), v[:, :3].amax(0)]) for v, _ in meshes])
    ids, xf = _instances(case["instances"], boxes, g)
    host = boxes.cpu().numpy()
    descs = [{"vertices": v, "triangles": t, "bounds": host[k]} for k, (v, t) in enumerate(meshes)]
    aabbs = torch.zeros(case["instances"], 6, device="cuda")
    descs.append({"aabbs": aabbs})
    n = int(sizes.sum()) + case["instances"]
    slots = 2 * n - (m + 1)
    return {"meshes": meshes, "boxes": boxes, "ids": ids, "xf": xf, "aabbs": aabbs, "descs": descs,
            "nodes": torch.zeros(slots * 8, dtype=torch.int32, device="cuda"),
            "lens": torch.zeros(slots, dtype=torch.int32, device="cuda"),
            "perm": torch.zeros(n, dtype=torch.int32, device="cuda")}


def _build_scene(ctx, s, stream):
    ctx.set_stream(stream.cuda_stream)
    instance_aabbs_device(ctx, s["boxes"], s["ids"], s["xf"], s["aabbs"])
    offs, _, _ = build_batch_device(ctx, BvhSettings(), s["descs"], s["nodes"], s["perm"], out_lens=s["lens"],
                                    stream=stream)
    return offs


def _prepare_train(case, g):
    b = case["batch"]
    # a trained network in the middle of its run: features of nodes are scale
    # free and of order one, a tenth of the nodes carry no position label
    x = torch.rand(b, 24, device="cuda", generator=g)
    label = torch.randint(0, 48, (b,), device="cuda", generator=g, dtype=torch.int32)
    label[torch.rand(b, device="cuda", generator=g) < 0.1] = -1
    gain = (torch.rand(b, device="cuda", generator=g) < 0.5).float()
    w = torch.from_numpy(learned.load_weights().view(np.int16)).cuda()
    n = w.shape[0]
    master = w.view(torch.bfloat16).float() * (1.0 + 1e-3 * torch.randn(n, device="cuda", generator=g))
    w = master.to(torch.bfloat16)
    return {"x": x, "label": label, "gain": gain, "w": w, "master": master,
            "m": 1e-3 * torch.randn(n, device="cuda", generator=g),
            "v": 1e-5 * (0.5 + torch.rand(n, device="cuda", generator=g)),
            "grad": torch.zeros(n, device="cuda"), "loss": torch.zeros(2, device="cuda")}


STEP, LEARNING_RATE, BETA1, BETA2, EPS = 1000, 1e-3, 0.9, 0.999, 1e-8


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "tlas_noalloc":
        lo = _uniform((case["n"], 3), -100.0, 100.0, g)
        s["aabbs"] = torch.cat([lo, lo + _uniform((case["n"], 3), 0.5, 8.0, g)], 1).contiguous()
        s["settings"] = BvhSettings().to_c(1, 1)
        s.update(_outputs(case["n"]))
    elif kind == "tlas_frame":
        lo = _uniform((case["meshes"], 3), -2.0, 0.0, g)
        s["boxes"] = torch.cat([lo, lo + _uniform((case["meshes"], 3), 0.2, 4.0, g)], 1).contiguous()
        s["ids"], s["xf"] = _instances(case["n"], s["boxes"], g)
        s["aabbs"] = torch.zeros(case["n"], 6, device="cuda")
        s["ctx"] = default_context()
        s.update(_outputs(case["n"]))
    elif kind in ("blas", "learned"):
        s["v"], s["t"] = _mesh(case["mesh"], case["n"], g)
        s["settings"] = _settings(case, _bounds(s["v"]))
        s["ctx"] = default_context()
        s.update(_outputs(s["t"].shape[0]))
        if kind == "learned":
            s["ctx"] = _lib.Context(0)
            s["ctx"].set_split_proposer(torch.from_numpy(learned.load_weights().view(np.int16)).cuda(), True)
            s["ctx"].set_proposer_gate(*learned.RECOMMENDED_GATE)
    elif kind == "batch":
        s.update(_scene(case, g))
        s["ctx"] = _lib.Context(0)
        s["ctx"].set_graph_capture(True)
        s["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()
    elif kind == "host":
        v, t = _icosphere_mesh(case["n"], g)
        s["v"], s["t"] = v.cpu().numpy(), t.cpu().numpy().view(np.uint32)
        s["settings"] = BvhSettings(name="mesh", bounds=_bounds(v))
    elif kind == "trace":
        v, t = _mesh("mixed", case["n"], g)
        n = t.shape[0]
        out = _outputs(n)
        torch.cuda.synchronize()  # the context builds on a stream of its own
        s["count"], _, _ = build_device(default_context(), BvhSettings(), out["nodes"], out["perm"], vertices=v,
                                        triangles=t, out_lens=out["lens"])
        s.update(out, v=v, t=t, rays=_rays(case["rays"], v.amin(0), v.amax(0), g),
                 hit_t=torch.zeros(case["rays"], device="cuda"),
                 hit_prim=torch.zeros(case["rays"], dtype=torch.int32, device="cuda"))
        tr = s["tracer"] = _lib.Tracer(0)
        tr.check(tr.L.mgbvh_tracer_set_blas_dev(tr.ptr, _vp(s["nodes"]), s["count"], None, _vp(v), 4 * v.shape[1],
                                                v.shape[0], _vp(t), _vp(s["perm"]), n, None))
        if case["wide"]:
            tr.check(tr.L.mgbvh_tracer_build_wide(tr.ptr, None, None))
    elif kind == "trace_scene":
        s.update(_scene(case, g))
        torch.cuda.synchronize()
        offs = _build_scene(default_context(), s, torch.cuda.current_stream())
        s["scene"] = Scene.from_batch(s["meshes"], offs, s["nodes"], None, s["perm"], s["ids"], s["xf"])
        s["tracer"] = _lib.Tracer(0)
        s["scene"].bind(s["tracer"])
        s["rays"] = _rays(case["rays"], s["aabbs"][:, :3].amin(0), s["aabbs"][:, 3:].amax(0), g)
    else:
        s.update(_prepare_train(case, g))
    return s


# ---------------------------------------------------------------- one pass

def _tree(s, count):
    """The caller's buffers; where leaves of several objects left the tree
    shorter than they are, the rows past it are cleared."""
    if count < s["lens"].shape[0]:
        s["nodes"][count * 8:].zero_()
        s["lens"][count:].zero_()
    return [s["nodes"], s["lens"], s["perm"]]


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "tlas_noalloc":
        L = _lib.load()
        count = ctypes.c_uint32(0)
        rc = L.mgbvh_build_aabbs_noalloc(_vp(s["aabbs"]), case["n"], ctypes.byref(s["settings"]), _vp(s["nodes"]),
                                         2 * case["n"] - 1, ctypes.byref(count), _vp(s["lens"]), _vp(s["perm"]),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc < 0:
            raise _lib.MgbvhError(rc, _lib.status_string(rc))
        return _tree(s, count.value)
    if kind == "tlas_frame":
        s["ctx"].set_stream(torch.cuda.current_stream().cuda_stream)
        instance_aabbs_device(s["ctx"], s["boxes"], s["ids"], s["xf"], s["aabbs"])
        count, _, _ = build_device(s["ctx"], BvhSettings(), s["nodes"], s["perm"], aabbs=s["aabbs"],
                                   out_lens=s["lens"])
        return [s["aabbs"]] + _tree(s, count)
    if kind in ("blas", "learned"):
        count, _, _ = build_device(s["ctx"], s["settings"], s["nodes"], s["perm"], vertices=s["v"],
                                   triangles=s["t"], out_lens=s["lens"], min_leaf_objects=case.get("min_leaf", 1),
                                   max_leaf_objects=case.get("max_leaf", 1))
        return _tree(s, count)
    if kind == "batch":
        offs = _build_scene(s["ctx"], s, s["stream"])
        return [s["aabbs"], torch.tensor(offs, dtype=torch.int64)] + _tree(s, offs[-1])
    if kind == "host":
        triangles = s["t"].copy()  # the caller's list, permuted in place by the call
        bvh = BoundingVolumeHierarchy.new(triangles, s["v"], s["settings"])
        return [bvh.nodes().view(np.uint32), bvh.lens, triangles]
    if kind == "trace":
        tr = s["tracer"]
        f = tr.L.mgbvh_trace_closest_wide_dev if case["wide"] else tr.L.mgbvh_trace_closest_dev
        tr.check(f(tr.ptr, _vp(s["rays"]), case["rays"], _vp(s["hit_t"]), _vp(s["hit_prim"]), None, None, None))
        return [s["hit_t"], s["hit_prim"]]
    if kind == "trace_scene":
        return list(trace_scene_device(s["tracer"], s["rays"])[:3])
    L = _lib.load()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    s["grad"].zero_()
    s["loss"].zero_()
    rc = L.mgbvh_mlp_train_step_dev(_vp(s["x"]), _vp(s["label"]), _vp(s["gain"]), case["batch"], _vp(s["w"]),
                                    _vp(s["grad"]), _vp(s["loss"]), stream)
    rc = rc or L.mgbvh_mlp_adam_dev(_vp(s["master"]), _vp(s["w"]), _vp(s["grad"]), _vp(s["m"]), _vp(s["v"]), STEP,
                                    LEARNING_RATE, BETA1, BETA2, EPS, stream)
    if rc:
        raise _lib.MgbvhError(rc, _lib.status_string(rc))
    return [s["grad"], s["loss"], s["master"], s["m"], s["v"], s["w"]]


# ---------------------------------------------------------------- what a pass cannot do without

def _tree_bytes(n):
    return 36 * (2 * n - 1) + 4 * n  # nodes and lens, permutation


def work(case):
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "tlas_noalloc":
        return {"bytes": 24 * n + _tree_bytes(n), "flops": 0}
    if kind == "tlas_frame":
        return {"bytes": 24 * case["meshes"] + 68 * n + 24 * n + _tree_bytes(n), "flops": 0}
    if kind in ("blas", "learned", "host"):
        # positions (unshared in the random and mixed meshes, half a vertex a
        # triangle on the icosphere) and index triples
        verts = n // 2 if case.get("mesh", "icosphere") == "icosphere" else 3 * n
        return {"bytes": 12 * verts + 12 * n + _tree_bytes(n), "flops": 0}
    if kind in ("batch", "trace_scene"):
        # the mean of a log-uniform size in [64, largest]
        total = int(case["meshes"] * (case["largest"] - 64) / math.log(case["largest"] / 64.0))
        if kind == "batch":
            return {"bytes": (12 + 21) * total + _tree_bytes(total + case["instances"]) + 92 * case["instances"],
                    "flops": 0}
        return {"bytes": case["rays"] * (32 + 12) + (64 + 48) * total + (64 + 80) * case["instances"], "flops": 0}
    if kind == "trace":
        return {"bytes": case["rays"] * (32 + 8) + (64 + 48) * n, "flops": 0}
    weights = 24 * 64 + 64 * 64 + 64 * 49
    b = case["batch"]
    # forward, weight gradients, and input gradients of the two upper layers
    return {"bytes": 104 * b + 8945 * (2 * 2 + 4 * 7), "flops": 2 * b * (2 * weights + 64 * 64 + 64 * 49)}


# ---------------------------------------------------------------- the same in 64 bits

def _exact_boxes(boxes, ids, xf):
    b, m = boxes.double()[ids.long()], xf.double().reshape(-1, 4, 4)  # [instance, column, row]
    p = []
    for c in range(8):
        x, y, z = b[:, 3 if c & 4 else 0], b[:, 4 if c & 2 else 1], b[:, 5 if c & 1 else 2]
        p.append(m[:, 0, :3] * x[:, None] + m[:, 1, :3] * y[:, None] + m[:, 2, :3] * z[:, None] + m[:, 3, :3])
    p = torch.stack(p)
    return torch.cat([p.amin(0), p.amax(0)], 1)


def _exact_train(case, seed):
    s = _prepare_train(case, _gen(seed))
    w = s["w"].double()
    shapes = ((64, 24), (64,), (64, 64), (64,), (49, 64), (49,))
    parts, at = [], 0
    for shape in shapes:
        size = math.prod(shape)
        parts.append(w[at:at + size].reshape(shape).clone().requires_grad_())
        at += size
    w1, b1, w2, b2, w3, b3 = parts
    gelu = torch.nn.functional.gelu
    out = gelu(gelu(s["x"].double() @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
    label = s["label"].long()
    ce = torch.nn.functional.cross_entropy(out[:, :48], label.clamp_min(0), reduction="none")
    ce = torch.where(label >= 0, ce, torch.zeros_like(ce))
    bce = torch.nn.functional.binary_cross_entropy_with_logits(out[:, 48], s["gain"].double(), reduction="none")
    ((ce + bce).sum() / case["batch"]).backward()
    grad = torch.cat([p.grad.reshape(-1) for p in parts])
    m = BETA1 * s["m"].double() + (1.0 - BETA1) * grad
    v = BETA2 * s["v"].double() + (1.0 - BETA2) * grad * grad
    master = s["master"].double() - LEARNING_RATE * (m / (1.0 - BETA1 ** STEP)) / (
        (v / (1.0 - BETA2 ** STEP)).sqrt() + EPS)
    return [grad, torch.stack([ce.sum(), bce.sum()]).detach(), master, m, v, None]


def exact(case, seed):
    """Instance boxes, gradients and updated weights. A tree is whole numbers
    (its bytes), and a hit's distance would need every triangle in 64 bits."""
    kind = case["kind"]
    if kind in ("tlas_frame", "batch"):
        s = prepare(case, seed) if kind == "tlas_frame" else _scene(case, _gen(seed))
        boxes = _exact_boxes(s["boxes"], s["ids"], s["xf"])
        return [boxes] + [None] * (3 if kind == "tlas_frame" else 4)
    if kind == "train":
        return _exact_train(case, seed)
    return None

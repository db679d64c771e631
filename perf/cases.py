"""The work that users of this library have it do, as measurable cases.

Five kinds of calls, each through the public entry points:

* ``render``  -- one frame: the Photon C API (clear, phRender, frame readback) or the flat scene ABI.
                 Scenes are the repository's own workloads (Cornell box, displaced GGX sphere, slit
                 room, many-light city) at their own and at smaller sizes.
* ``guided``  -- a frame rendered with path guiding, the network starting untrained and learning
                 during the render, as the first render of a scene does.
* ``batch``   -- many scenes rendered as one wavefront, every frame read back.
* ``query``   -- closest-hit and occlusion queries on a triangle mesh, with host rays (as a picking or
                 collision tool calls them) or rays and hits resident on the GPU (as a tracer does).
* ``guide``   -- the path-guiding network on its own: mixtures at query points (forward), a loss
                 gradient (backward), a run of Adam steps (training).

``work`` counts each input and output once; the operations are the box and triangle tests of the
rays a render traces on average (per scene, as the benchmark counts them), or the network's own
multiply-adds.
"""

import ctypes
import functools
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "photon-v2_b200"))

import photon_gpu  # noqa: E402
import scenes  # noqa: E402

ESTIMATORS = {"bneept": photon_gpu.BNEEPT, "bvpt": photon_gpu.BVPT, "bvptdl": photon_gpu.BVPTDL}
# traced rays per path (closest + shadow), and operations per ray: 7 nodes of 8 boxes, 5 triangles
RAYS_PER_PATH = {"cornell": 9.0, "cornell_glossy": 9.0, "sphere": 4.3, "slit_room": 9.3, "city": 6.0}
FLOPS_PER_RAY = 7 * 8 * 12 + 5 * 60
# bytes a triangle takes in the tree: its 48-byte record and its share of the 80-byte nodes
BYTES_PER_TRI = 48 + 14
GUIDE_PARAMS = 29480
GUIDE_FLOPS = 58368   # one query forward


def listed():
    return [
        # a thumbnail of the Cornell box, redrawn while a user drags something: latency
        {"name": "thumbnail", "kind": "render", "api": "c", "scene": "cornell", "size": 0, "width": 64, "height": 48,
         "spp": 1, "depth": 8, "estimator": "bneept", "filter": "box"},
        # the Cornell box configuration: 256 x 256, 64 samples, depth 8, through the C API
        {"name": "cornell", "kind": "render", "api": "c", "scene": "cornell", "size": 0, "width": 256, "height": 256,
         "spp": 64, "depth": 8, "estimator": "bneept", "filter": "box"},
        # a scene file that names no filter (Blackman-Harris then) under a sky dome, odd frame size
        {"name": "default_filter", "kind": "render", "api": "c", "scene": "cornell_glossy", "size": 0, "width": 637,
         "height": 359, "spp": 32, "depth": 10, "estimator": "bneept", "filter": "bh"},
        # the benchmarked 1.3 M-triangle GGX scene at 1024 x 1024, a sixteenth of its samples
        {"name": "ggx_1m", "kind": "render", "api": "flat", "scene": "sphere", "size": 8, "width": 1024, "height": 1024,
         "spp": 16, "depth": 10, "estimator": "bneept", "filter": "box"},
        # the slit room (2 M triangles, a third of them glass) at 1024 x 1024, a progressive pass
        {"name": "slit_room", "kind": "render", "api": "flat", "scene": "slit_room", "size": 166667, "width": 1024,
         "height": 1024, "spp": 2, "depth": 10, "estimator": "bneept", "filter": "box"},
        # a quarter-scale many-light city at 1920 x 1080
        {"name": "city", "kind": "render", "api": "flat", "scene": "city", "size": 110, "width": 1920, "height": 1080,
         "spp": 8, "depth": 12, "estimator": "bneept", "filter": "box"},
        # a render whose guiding network learns while it renders
        {"name": "guided", "kind": "guided", "api": "flat", "scene": "cornell", "size": 0, "width": 256, "height": 256,
         "spp": 192, "depth": 8, "estimator": "bneept", "filter": "box"},
        # many small jobs as one wavefront (the batched workload's scenes at an eighth of their samples)
        {"name": "batch", "kind": "batch", "first": 0, "count": 8, "divisor": 8, "depth": 10},
        # a tool that asks for a handful of hits: latency of the host entry points
        {"name": "pick", "kind": "query", "where": "host", "boxes": 2000, "rays": 1000},
        # device-resident incoherent rays against 2 M triangles: throughput
        {"name": "trace", "kind": "query", "where": "device", "boxes": 166667, "rays": 4000000},
        # guiding mixtures at the vertices of a frame tile
        {"name": "guide_mixture", "kind": "guide", "do": "mixture", "n": 100000, "steps": 1, "batch": 0},
        # guiding network fitted to recorded samples: the default batch, 32 Adam steps
        {"name": "guide_train", "kind": "guide", "do": "train", "n": 131072, "steps": 32, "batch": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.55:
        scene = rng.choice(["cornell", "cornell", "cornell_glossy", "sphere", "slit_room", "city"])
        size = {"cornell": 0, "cornell_glossy": 0, "sphere": rng.choice([3, 4, 5, 6, 7]),
                "slit_room": _log(rng, 100, 150000), "city": _log(rng, 8, 100)}[scene]
        width, height = _log(rng, 32, 1280), _log(rng, 32, 1024)
        most = max(1.0, min(256.0, 16e6 / (width * height)))
        return {"kind": "render", "api": rng.choice(["c", "flat"]) if scene in ("cornell", "cornell_glossy") else "flat",
                "scene": scene, "size": size, "width": width, "height": height, "spp": _log(rng, 1, most),
                "depth": rng.choice([1, 3, 6, 8, 10, 12, 10000]) if scene != "slit_room" else rng.choice([2, 6, 10]),
                "estimator": rng.choice(["bneept", "bneept", "bneept", "bvpt", "bvptdl"]),
                "filter": rng.choice(["box", "box", "gaussian", "mn", "bh"])}
    if pick < 0.60:
        return {"kind": "guided", "api": "flat", "scene": "cornell", "size": 0, "width": _log(rng, 128, 400),
                "height": _log(rng, 128, 400), "spp": _log(rng, 64, 96), "depth": rng.choice([4, 8]),
                "estimator": "bneept", "filter": "box"}
    if pick < 0.66:
        return {"kind": "batch", "first": rng.randint(0, 63), "count": rng.randint(2, 8),
                "divisor": rng.choice([16, 64]), "depth": rng.choice([4, 10])}
    if pick < 0.82:
        return {"kind": "query", "where": rng.choice(["host", "device"]), "boxes": _log(rng, 3, 160000),
                "rays": _log(rng, 1, 3000000)}
    do = rng.choice(["mixture", "gradient", "train"])
    n = _log(rng, 1 if do == "mixture" else 100, 400000)
    return {"kind": "guide", "do": do, "n": n, "steps": rng.randint(2, 24) if do == "train" else 1,
            "batch": min(n, _log(rng, 64, 65536)) if do == "train" else 0}


class _Held:
    """What a program holds between calls; the library's objects are closed with it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)
        self.objects = kw.get("objects", [])

    def __del__(self):
        for o in self.objects:
            try:
                o.close()
            except Exception:
                pass


# ---------------------------------------------------------------------------------------------
# inputs

@functools.lru_cache(maxsize=None)
def _sphere_asset(level):
    """The displaced sphere's triangles, a fixed asset of the workload (seconds to displace in NumPy)."""
    return scenes.ggx_sphere(level)


def _scene(case, seed):
    """The workload's scene seen from a camera, and with light and surface values, of this seed."""
    rng = np.random.default_rng(seed)
    args = dict(width=case["width"], height=case["height"], spp=case["spp"], max_bounces=case["depth"],
                estimator=case["estimator"])
    name = case["scene"]
    if name == "cornell":
        sc = scenes.cornell(**args)
    elif name == "cornell_glossy":
        sc = scenes.cornell_glossy(**args)
        sc.env_image = scenes.sky_image(seed=int(rng.integers(1 << 20)))
    elif name == "sphere":
        base = _sphere_asset(case["size"])
        sc = scenes.Scene(base.name, args["width"], args["height"], args["spp"], args["max_bounces"], base.cam_pos,
                          base.cam_dir, base.cam_up, base.fov_deg, list(base.groups), estimator=args["estimator"],
                          env_radiance=base.env_radiance)
        for i, g in enumerate(sc.groups):
            if g.material.kind == "conductor":
                sc.groups[i] = scenes.MeshGroup(g.tris, scenes.Material(
                    "conductor", roughness=float(rng.uniform(0.05, 0.5)),
                    f0=tuple(float(x) for x in rng.uniform(0.5, 1.0, 3))))
        a = float(rng.uniform(-0.6, 0.6))   # orbit the camera around the sphere
        sc.cam_pos = (4.2 * math.sin(a), 1.6, -4.2 * math.cos(a))
        sc.cam_dir = (-math.sin(a), -0.12, math.cos(a))
    elif name == "slit_room":
        sc = scenes.slit_room(num_boxes=case["size"], seed=int(rng.integers(1 << 20)), **args)
    else:
        blocks = case["size"]
        sc = scenes.city(blocks=blocks, num_lights=max(4, min(1000, blocks * blocks // 10)),
                         seed=int(rng.integers(1 << 20)), **args)
    sc.sample_filter = case["filter"]
    k = float(rng.uniform(0.7, 1.3))
    for i, g in enumerate(sc.groups):
        if g.radiance is not None:
            sc.groups[i] = scenes.MeshGroup(g.tris, g.material, tuple(float(x) * k for x in g.radiance))
    return sc


def _rays(lo, hi, n, seed):
    """Half coherent rays from one viewpoint, half with random origins and directions, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    lo = torch.tensor(lo, device="cuda", dtype=torch.float32)
    ext = torch.tensor(hi, device="cuda", dtype=torch.float32) - lo
    o = lo + ext * torch.rand(n, 3, device="cuda", generator=g)
    d = torch.randn(n, 3, device="cuda", generator=g)
    view = n // 2
    o[:view] = lo + ext * torch.tensor([0.1, 0.55, 0.1], device="cuda")
    side = max(1, int(math.isqrt(max(1, view))))
    i = torch.arange(view, device="cuda")
    d[:view, 0] = 0.55 + 0.9 * ((i % side).float() + torch.rand(view, device="cuda", generator=g)) / side - 0.45
    d[:view, 1] = -0.15 + 0.9 * ((i // side).float() + torch.rand(view, device="cuda", generator=g)) / (side + 1) - 0.45
    d[:view, 2] = 0.8
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.empty(n, 8, device="cuda")
    rays[:, :3], rays[:, 3], rays[:, 4:7], rays[:, 7] = o, 0.0, d, 1e30
    return rays


def _query_mesh(boxes, seed):
    """A room of `boxes` random boxes (the slit room's geometry)."""
    sc = scenes.slit_room(num_boxes=boxes, seed=int(seed) % (1 << 20))
    return np.concatenate([g.tris for g in sc.groups])


def _guide_params(rng):
    """He-initialised weights and small biases in the packed order."""
    parts = []
    for fan_in, fan_out, scale in ((224, 64, 1.0), (64, 64, 1.0), (64, 64, 1.0), (64, 64, 1.0), (64, 40, 0.3)):
        parts.append(rng.normal(0.0, math.sqrt(2.0 / fan_in) * scale, fan_in * fan_out))
        parts.append(rng.normal(0.0, 0.1, fan_out))
    return np.concatenate(parts).astype(np.float32)


def _guide_inputs(case, seed):
    """Query features; for training also directions around a position-dependent mean, and weights."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    params = _guide_params(rng)
    feat = rng.random((n, 7), dtype=np.float32)
    mu = np.stack([feat[:, 0] - 0.5, feat[:, 1] - 0.5, np.full(n, 0.3, np.float32)], axis=1)
    d = mu / np.linalg.norm(mu, axis=1, keepdims=True) + 0.3 * rng.standard_normal((n, 3), dtype=np.float32)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    w = np.exp(rng.standard_normal(n, dtype=np.float32))
    return params, feat, d, w


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("render", "guided"):
        sc = _scene(case, seed)
        if case["api"] == "c":
            eng = photon_gpu.PhotonEngine()
            with tempfile.TemporaryDirectory() as tmp:
                with open(os.path.join(tmp, "scene.p2"), "w") as f:
                    f.write(scenes.to_sdl(sc, mesh_format="ply"))
                scenes.write_meshes(sc, tmp)
                scenes.write_env(sc, tmp)
                eng.set_working_directory(tmp)
                if not eng.load_file(os.path.join(tmp, "scene.p2")):
                    raise RuntimeError(eng.errors())
                eng.set_max_bounces(sc.max_bounces)
                eng.set_seed(seed)
                eng.update()
            return _Held(case=case, objects=[eng])
        sc.env_image = None   # the flat scene ABI takes constant environments
        rs = photon_gpu.RenderScene(sc)
        if case["filter"] != "box":
            rs.set_filter(case["filter"])
        if kind == "guided":
            rs.set_guiding(True, True)
        return _Held(case=case, seed=int(seed), objects=[rs])
    if kind == "batch":
        rng = np.random.default_rng(seed)
        scs = [scenes.batch_scene((case["first"] + i) % 64, case["depth"]) for i in range(case["count"])]
        for sc in scs:   # every job seen from its own side
            a = float(rng.uniform(0.0, 2 * math.pi))
            sc.cam_pos, sc.cam_dir = (tuple(x * math.cos(a) + z * math.sin(a) if i == 0 else y if i == 1
                                            else z * math.cos(a) - x * math.sin(a) for i in range(3))
                                      for x, y, z in (sc.cam_pos, sc.cam_dir))
        return _Held(case=case, seed=int(seed), spp=[max(1, s.spp // case["divisor"]) for s in scs],
                     objects=[photon_gpu.RenderScene(s) for s in scs])
    if kind == "query":
        tris = _query_mesh(case["boxes"], seed)
        geo = photon_gpu.Geometry(tris)
        n = case["rays"]
        rays = _rays(tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0), n, seed)
        if case["where"] == "host":
            return _Held(case=case, objects=[geo], rays=rays.cpu().numpy())
        # the leaf triangle a device hit names, as a primitive index of the caller's mesh (last: a miss)
        prim = np.append(geo.export()[1]["prim"].astype(np.int32), np.int32(-1))
        return _Held(case=case, objects=[geo], rays=rays, prim=torch.from_numpy(prim).cuda(),
                     hits=torch.empty(n, 2, device="cuda", dtype=torch.int32),
                     occluded=torch.empty(n, device="cuda", dtype=torch.int32))
    params, feat, d, w = _guide_inputs(case, seed)
    return _Held(case=case, params=params, feat=feat, dirs=d, weights=w)


# ---------------------------------------------------------------------------------------------
# the calls

def run(state):
    case = state.case
    kind = case["kind"]
    if kind in ("render", "guided"):
        if case["api"] == "c":
            eng = state.objects[0]
            eng.clear_film()
            eng.render()
            return eng.frame()
        rs = state.objects[0]
        rs.clear()
        if kind == "guided":
            rs.guide_reset()
        rs.render(case["spp"], max_bounces=case["depth"], estimator=ESTIMATORS[case["estimator"]], seed=state.seed)
        return rs.film(with_sums=False)[0]
    if kind == "batch":
        for rs in state.objects:
            rs.clear()
        photon_gpu.render_scenes_wavefront(state.objects, state.spp, max_bounces=case["depth"], seed=state.seed)
        return [rs.film(with_sums=False)[0] for rs in state.objects]
    if kind == "query":
        geo = state.objects[0]
        if case["where"] == "host":
            prim, t, bary = geo.closest(state.rays)
            return {"prim": prim, "t": t, "bary": bary, "occluded": geo.occluded(state.rays)}
        lib = photon_gpu.load()
        rays, n = ctypes.c_void_p(state.rays.data_ptr()), case["rays"]
        status = lib.pgpu_trace_closest_device(geo.id, rays, n, ctypes.c_void_p(state.hits.data_ptr()), None)
        status = status or lib.pgpu_trace_any_device(geo.id, rays, n, ctypes.c_void_p(state.occluded.data_ptr()), None)
        if status:
            raise RuntimeError(lib.pgpu_last_error().decode())
        leaf = state.hits[:, 0]
        prim = state.prim[torch.where(leaf < 0, state.prim.numel() - 1, leaf)]   # a miss is 0xFFFFFFFF
        return {"prim": prim, "t": state.hits.view(torch.float32)[:, 1], "occluded": state.occluded}
    if case["do"] == "mixture":
        return photon_gpu.guide_mixture(state.params, state.feat)
    if case["do"] == "gradient":
        return photon_gpu.guide_gradients(state.params, state.feat, state.dirs, state.weights)
    return photon_gpu.guide_train(state.params, state.feat, state.dirs, state.weights, case["steps"], case["batch"],
                                  lr=1e-3)


def _triangles(case):
    if case["scene"] == "sphere":
        return 20 * 4 ** case["size"] + 6
    return {"cornell": 36, "cornell_glossy": 36, "slit_room": 12 * case["size"], "city": 108 * case["size"] ** 2}[case["scene"]]


def work(case):
    kind = case["kind"]
    if kind in ("render", "guided"):
        pixels = case["width"] * case["height"]
        if case["estimator"] == "bvptdl" or case["depth"] == 1:
            rays = 2.0
        else:
            rays = min(RAYS_PER_PATH[case["scene"]], 2.0 * case["depth"])
        return {"bytes": BYTES_PER_TRI * _triangles(case) + 12.0 * pixels,
                "flops": float(pixels) * case["spp"] * rays * FLOPS_PER_RAY}
    if kind == "batch":   # its scenes average 217,000 triangles, 0.42 M pixels and 136 samples
        return {"bytes": case["count"] * (BYTES_PER_TRI * 2.17e5 + 12.0 * 4.2e5),
                "flops": case["count"] * 4.2e5 * 136 / case["divisor"] * 5.0 * FLOPS_PER_RAY}
    if kind == "query":   # two queries per ray; prim, t (host: barycentrics) and the occlusion flag out
        out = 24 if case["where"] == "host" else 12
        return {"bytes": 12.0 * case["boxes"] * BYTES_PER_TRI + (2 * 32.0 + out) * case["rays"],
                "flops": 2.0 * case["rays"] * FLOPS_PER_RAY}
    if case["do"] == "mixture":
        return {"bytes": 4.0 * GUIDE_PARAMS + case["n"] * (28.0 + 192.0), "flops": float(case["n"]) * GUIDE_FLOPS}
    rows = case["n"] if case["do"] == "gradient" else case["steps"] * case["batch"]
    return {"bytes": 8.0 * GUIDE_PARAMS + 44.0 * case["n"], "flops": 3.0 * rows * GUIDE_FLOPS}


# ---------------------------------------------------------------------------------------------
# the same answers in 64 bits

def _mlp64(params, feat):
    """Raw outputs [n, 8, 5] of the network for FP64 parameters (a list) and features."""
    c = (torch.arange(32, device="cuda", dtype=torch.float64) + 0.5) / 32
    x = torch.exp(-0.5 * ((feat[:, :, None] - c) * 32) ** 2).reshape(feat.shape[0], 224)
    for layer in range(5):
        x = x @ params[2 * layer] + params[2 * layer + 1]
        if layer < 4:
            x = torch.relu(x)
    return x.reshape(-1, 8, 5)


def _mixture64(raw):
    w = torch.softmax(raw[:, :, 0], dim=1)
    m = raw[:, :, 1:4]
    mu = m / m.norm(dim=2, keepdim=True)
    kappa = raw[:, :, 4].exp().clamp(1e-2, 5e3)
    return w, mu, kappa


def _params64(flat):
    out, at = [], 0
    p = torch.as_tensor(flat, device="cuda").double()
    for a, b in ((224, 64), (64, 64), (64, 64), (64, 64), (64, 40)):
        out += [p[at:at + a * b].reshape(a, b), p[at + a * b:at + a * b + b]]
        at += a * b + b
    return out


def _loss64(params, feat, d, w):
    pi, mu, kappa = _mixture64(_mlp64(params, feat))
    log_v = torch.log(kappa / (2 * math.pi * (1 - torch.exp(-2 * kappa)))) + kappa * ((mu * d[:, None, :]).sum(-1) - 1)
    return -(w * torch.logsumexp(torch.log(pi) + log_v, dim=1)).sum() / w.sum()


def _exact_guide(case, seed):
    flat, feat, d, w = _guide_inputs(case, seed)
    feat, d, w = (torch.as_tensor(a, device="cuda").double() for a in (feat, d, w))
    params = _params64(flat)
    if case["do"] == "mixture":
        out = torch.empty(case["n"], 8, 6, device="cuda", dtype=torch.float64)
        for at in range(0, case["n"], 65536):
            pi, mu, kappa = _mixture64(_mlp64(params, feat[at:at + 65536]))
            c = pi * kappa / (2 * math.pi * (1 - torch.exp(-2 * kappa)))
            out[at:at + 65536] = torch.cat([pi[..., None], mu, kappa[..., None], c[..., None]], dim=2)
        return out
    for p in params:
        p.requires_grad_(True)

    def gradient(rows):
        """Loss and gradient of the batch, in pieces that fit."""
        total, loss, grads = w[rows].sum(), 0.0, [torch.zeros_like(p) for p in params]
        index = torch.arange(rows.start, rows.stop, device="cuda")
        for part in index.split(65536):
            piece = _loss64(params, feat[part], d[part], w[part]) * (w[part].sum() / total)
            for g, e in zip(grads, torch.autograd.grad(piece, params)):
                g += e
            loss += float(piece.detach())
        return loss, grads

    if case["do"] == "gradient":
        loss, grads = gradient(slice(0, case["n"]))
        return loss, torch.cat([g.reshape(-1) for g in grads])
    n, batch = case["n"], min(case["batch"], case["n"])
    m, v, losses = [torch.zeros_like(p) for p in params], [torch.zeros_like(p) for p in params], []
    for step in range(case["steps"]):
        first = step * batch % n
        loss, grads = gradient(slice(first, first + min(batch, n - first)))
        losses.append(loss)
        with torch.no_grad():
            for p, g, a, b in zip(params, grads, m, v):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).add_(g * g, alpha=0.001)
                p -= 1e-3 * (a / (1 - 0.9 ** (step + 1))) / ((b / (1 - 0.999 ** (step + 1))).sqrt() + 1e-8)
    return torch.cat([p.detach().reshape(-1) for p in params]), torch.tensor(losses, dtype=torch.float64)


def _exact_query(case, seed):
    """Brute force over every triangle: distances and barycentrics of the closest hits."""
    tris_np = _query_mesh(case["boxes"], seed)
    rays = _rays(tris_np.reshape(-1, 3).min(0), tris_np.reshape(-1, 3).max(0), case["rays"], seed).double()
    tris = torch.from_numpy(tris_np).cuda().double()
    a, e1, e2 = tris[:, 0], tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]
    normal = torch.linalg.cross(e1, e2)
    t_all = torch.zeros(rays.shape[0], device="cuda", dtype=torch.float64)
    bary = torch.zeros(rays.shape[0], 3, device="cuda", dtype=torch.float64)
    step = max(1, int(2e7) // tris.shape[0])
    for at in range(0, rays.shape[0], step):
        o, d = rays[at:at + step, None, :3], rays[at:at + step, None, 4:7]
        s = o - a
        den = -(d * normal).sum(-1)
        q = torch.linalg.cross(s, d.expand_as(s))
        u, v = (e2 * q).sum(-1) / den, -(e1 * q).sum(-1) / den
        t = (s * normal).sum(-1) / den
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0) & (t <= 1e30), t, math.inf)
        best, k = t.min(dim=1)
        hit = torch.isfinite(best)
        bu, bv = u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]
        t_all[at:at + step] = torch.where(hit, best, 0.0)
        bary[at:at + step] = torch.where(hit[:, None], torch.stack([1 - bu - bv, bu, bv], dim=1), 0.0)
    return t_all, bary


def exact(case, seed):
    if case["kind"] == "guide":
        return _exact_guide(case, seed)
    if case["kind"] == "query" and case["rays"] * (12 * case["boxes"] + 20) <= 4e9:
        t, bary = _exact_query(case, seed)
        if case["where"] == "host":
            return {"prim": None, "t": t, "bary": bary, "occluded": None}
        # a device miss reports t = 0 as well
        return {"prim": None, "t": t, "occluded": None}
    return None   # renders (no 64-bit path tracer without this repository's code) and the largest queries

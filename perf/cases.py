"""The calls that users of this path tracer make, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes what a program has in
hand before the call (scene, tree, device context, host buffers), ``run``
makes the call through the package's public classes and returns its results.

Kinds of case:

  frame   one rendered picture of a scene: PathTracer.render() of `spp`
          passes with the accumulation restarted by a camera set, then
          getFrameBuffer() into a host buffer the program keeps (pinned, as
          the benchmark's end-to-end figure has it)
  batch   the same for several scenes through Batch (one launch)
  rays    traceRays(): closest hits of a list of host rays
  infer   RadianceCache.infer(): the network's outputs for host inputs
  grads   RadianceCache.gradients(): loss and weight gradients
  jpeg    read_jpeg(): a texture file's bytes to RGBA8
  load    a scene into a render context: Bvh() and Renderer()
"""
import math

import numpy as np
import torch

from zig_ornament_gb300 import _lib, ornament, scenes, textures

KERNELS = {"mega": _lib.KERNEL_MEGA, "wavefront": _lib.KERNEL_WAVEFRONT, "cached": _lib.KERNEL_CACHED,
           "cached_wavefront": _lib.KERNEL_CACHED_WAVEFRONT}
SEMANTICS = {"hip": _lib.SEMANTICS_HIP, "wgsl": _lib.SEMANTICS_WGSL}

FRAME = dict(kind="frame", kernel="mega", semantics="hip", tree="reference", watertight=False, flip=False, gamma=1.0,
             streams=0)


def listed():
    return [
        # an interactive viewport of a small scene: one pass per camera move;
        # latency and launches are what it costs
        dict(FRAME, name="preview_96x64", scene="small", width=96, height=64, spp=1, depth=8),
        # the sphere field at its configuration's resolution, samples and depth
        dict(FRAME, name="spheres_640x360", scene="spheres", width=640, height=360, spp=64, depth=10),
        # the headline scene at its resolution, a quarter of its samples
        dict(FRAME, name="instanced_1080p", scene="instanced", width=1920, height=1080, spp=64, depth=8),
        # many instances of glass, metal and textured meshes, long paths, odd size
        dict(FRAME, name="large_1279x719", scene="large", width=1279, height=719, spp=8, depth=16),
        # the wavefront kernel with the shader backend's semantics, gamma and flip, ragged size
        dict(FRAME, name="wavefront_wgsl_1001x563", scene="instanced", width=1001, height=563, spp=16, depth=8,
             kernel="wavefront", semantics="wgsl", flip=True, gamma=2.2),
        # light sampling without cache queries (every path a training path), eight sample streams per pixel
        dict(FRAME, name="light_sampling_640x360", scene="room", width=640, height=360, spp=1, depth=8, kernel="cached",
             streams=8),
        # several scenes of uneven size in one launch
        dict(name="batch_6", kind="batch", count=6, width=1280, spp=16, tris=50_000),
        # a host program's ray queries against a scene
        dict(name="rays_200k", kind="rays", scene="instanced", n=200_000, visits=False),
        # the cache's network alone: forward over an odd number of samples, and one batch's gradients
        dict(name="infer_100003", kind="infer", n=100_003),
        dict(name="grads_16384", kind="grads", n=16_384),
        # a planet texture of the example program's size
        dict(name="jpeg_2048x1024", kind="jpeg", width=2048, height=1024, flip=True),
        # a scene of 281 k triangles from arrays to a context that can render
        dict(name="load_lbvh_282k", kind="load", meshes=8, freq=42, instances=256, tree="lbvh"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# most samples per frame, so that no frame costs more than the largest listed one
SAMPLES = {"small": 60e6, "spheres": 60e6, "instanced": 30e6, "large": 6e6, "room": 20e6}


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["batch", "rays", "rays", "infer", "grads", "jpeg", "load"])
    if kind == "frame":
        c = dict(FRAME, scene=rng.choice(["small", "spheres", "instanced", "instanced", "large", "room"]))
        c["width"] = _log(rng, 64, 1920)
        c["height"] = max(33, int(c["width"] * rng.uniform(0.5, 0.8)))
        c["kernel"] = rng.choice(["mega"] * 4 + ["wavefront"] * 2 + ["cached", "cached_wavefront"])
        cached = c["kernel"].startswith("cached")
        c["streams"] = rng.choice([1, 4, 8]) if cached else 0
        most = SAMPLES[c["scene"]] / (c["width"] * c["height"]) / (4 * c["streams"] if cached else 1)
        c["spp"] = max(1, min(_log(rng, 1, 128), int(most)))
        if cached:
            c["streams"] = min(c["streams"], max(1, int(4 * most)))
            c["spp"] = min(c["spp"], 2)
        c["depth"] = rng.randint(2, 16)
        c["semantics"] = rng.choice(["hip", "hip", "wgsl"])
        c["tree"] = rng.choice(["reference", "reference", "sah"])
        c["watertight"] = rng.random() < 0.15
        c["flip"] = rng.random() < 0.5
        c["gamma"] = rng.choice([1.0, 2.2])
        return c
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 8), width=_log(rng, 200, 1280), spp=_log(rng, 2, 24),
                    tris=_log(rng, 1_000, 100_000))
    if kind == "rays":
        return dict(kind=kind, scene=rng.choice(["small", "spheres", "instanced", "large"]), n=_log(rng, 1, 1_000_000),
                    visits=rng.random() < 0.3)
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 1, 400_000))
    if kind == "grads":
        return dict(kind=kind, n=_log(rng, 100, 60_000))
    if kind == "jpeg":
        return dict(kind=kind, width=_log(rng, 17, 2048), height=_log(rng, 9, 1024), flip=rng.random() < 0.7)
    return dict(kind=kind, meshes=rng.randint(1, 16), freq=rng.randint(3, 50), instances=_log(rng, 1, 1000),
                tree=rng.choice(["lbvh", "lbvh", "reference"]))


# ---- inputs -------------------------------------------------------------------------------------


def _scene(name, width, height, seed):
    if name == "small":
        return scenes.small_test_scene(width, height, seed=seed)
    if name == "spheres":
        return scenes.spheres_scene(width, height, seed=seed)
    if name == "instanced":
        return scenes.instanced_meshes_scene(width, height, seed=seed, texture_size=256)
    if name == "large":
        return scenes.large_scene(width, height, seed=seed, n_instances=1024, total_tris=1_000_000, texture_size=256)
    return scenes.cornell_box_scene(width, height, light_radiance=4.0 + seed % 97 / 12.0)


def _load_scene(case, seed):
    """Geodesic meshes with a bumpy surface, and instances of them."""
    rs = np.random.default_rng(seed)
    scene = ornament.Scene()
    v, n, uv, idx = scenes.icosphere(case["freq"])
    meshes = []

    def placed():
        move = ornament.translation(*rs.uniform(-50, 50, 3))
        size = ornament.scaling(*[float(rs.uniform(0.5, 3.0))] * 3)
        return ornament.mul(ornament.mul(size, scenes.random_rotation(rs)), move)

    for _ in range(case["meshes"]):
        bumpy = v.copy()
        bumpy[:, :3] *= (4.0 + 0.3 * np.sin(v[:, :3] @ rs.uniform(-9, 9, 3)) + 0.3 * np.cos(v[:, :3] @ rs.uniform(-9, 9, 3)))[:, None]
        mesh = scene.createMesh(bumpy, idx, n, idx, uv, idx, placed(), scenes.random_material(scene, rs))
        scene.attachMesh(mesh)
        meshes.append(mesh)
    for i in range(case["instances"]):
        scene.attachMeshInstance(scene.createMeshInstance(meshes[i % len(meshes)], placed(), scenes.random_material(scene, rs)))
    return scene


def _batch_scenes(case, seed):
    """(scene, width, height, spp) of uneven triangle counts, instances, sizes and samples."""
    for i in range(case["count"]):
        share = (1.0, 0.4, 0.15, 0.7)[i % 4]
        w = max(64, int(case["width"] * (1.0, 0.5, 0.2)[i % 3]))
        tris = case["tris"] * share
        scene = scenes.instanced_meshes_scene(w, w * 9 // 16, seed=seed + i, n_blas=1 + i % 4, n_instances=4 << (i % 6),
                                              tri_range=(tris * 0.8, tris * 1.25), n_textures=2, texture_size=256)
        yield scene, w, w * 9 // 16, max(1, int(case["spp"] * (1.0, 0.25, 4.0)[i % 3]))


def _host_frame(width, height):
    """The program's frame, pinned: (array, the tensor that owns its memory)."""
    owner = torch.empty((width * height, 4), dtype=torch.float32, pin_memory=torch.cuda.is_available())
    return owner.numpy(), owner


def _set_state(state, case):
    state.setDepth(case["depth"])
    state.setIterations(case["spp"])
    state.setFlipY(case["flip"])
    state.setGamma(case["gamma"])
    state.kernel = KERNELS[case["kernel"]]
    state.semantics = SEMANTICS[case["semantics"]]
    state.triangle_test = _lib.TRIANGLE_WATERTIGHT if case["watertight"] else _lib.TRIANGLE_MOLLER_TRUMBORE
    if case["kernel"].startswith("cached"):
        state.spp_per_launch = case["streams"]
        state.sampler = _lib.SAMPLER_SOBOL


def _mlp_weights(rs):
    """He-uniform weights in the cache's order (output rows 3..15 are padding)."""
    shapes = [(64, 256)] + [(64, 64)] * 4 + [(16, 64)]
    w = [rs.uniform(-1, 1, s) * math.sqrt(6.0 / s[1]) for s in shapes]
    w[-1][3:] = 0.0
    return [m.astype(np.float32) for m in w]


def _mlp_inputs(case, seed):
    rs = np.random.default_rng(seed)
    weights = _mlp_weights(rs)
    x = rs.random((case["n"], 10), dtype=np.float32)
    x[:, 9] = np.where(rs.random(case["n"]) < 0.7, np.float32(1.0), x[:, 9])   # lambertian surfaces: roughness 1
    target = rs.exponential(0.5, (case["n"], 3)).astype(np.float32)
    target[rs.random(case["n"]) < 0.05] = -1.0                                   # paths without a cache vertex
    return weights, x, target


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "frame":
        w, h = case["width"], case["height"]
        scene = _scene(case["scene"], w, h, seed)
        pt = ornament.PathTracer(scene, bvh=ornament.Bvh(scene, builder=case["tree"]))
        _set_state(pt.state, case)
        pt.setResolution(ornament.Resolution(w, h))
        if case["kernel"].startswith("cached"):
            s["cache"] = ornament.RadianceCache(seed=1 + seed % 1000, train_shift=0)
            pt.renderer.attach_cache(s["cache"])
        s["pt"] = pt
        s["dst"], s["owner"] = _host_frame(w, h)
    elif kind == "batch":
        s["renderers"], s["scenes"], s["dst"], s["owner"] = [], [], [], []
        for scene, w, h, spp in _batch_scenes(case, seed):
            r = ornament.Renderer(ornament.Bvh(scene))
            state = ornament.State()
            state.setDepth(8)
            state.setIterations(spp)
            r.set_state(state.to_struct())
            r.set_resolution(w, h)
            s["renderers"].append(r)
            s["scenes"].append(scene)
            dst, owner = _host_frame(w, h)
            s["dst"].append(dst)
            s["owner"].append(owner)
        s["batch"] = ornament.Batch(s["renderers"])
    elif kind == "rays":
        scene = _scene(case["scene"], 640, 360, seed)
        s["pt"] = ornament.PathTracer(scene)
        rs = np.random.default_rng(seed)
        extent = {"small": 6.0, "spheres": 12.0, "instanced": 60.0, "large": 140.0}[case["scene"]]
        s["rays"] = np.concatenate([rs.uniform(-extent, extent, (case["n"], 3)), rs.normal(size=(case["n"], 3))],
                                   1).astype(np.float32)
        s["visits"] = case["visits"]
    elif kind in ("infer", "grads"):
        weights, s["x"], s["target"] = _mlp_inputs(case, seed)
        s["cache"] = ornament.RadianceCache(seed=1)
        s["cache"].set_params(np.concatenate([m.ravel() for m in weights]))
    elif kind == "jpeg":
        s["file"] = _jpeg_file(case["width"], case["height"], seed)
        s["flip"] = case["flip"]
    else:
        s["scene"] = _load_scene(case, seed)
        s["tree"] = case["tree"]
    return s


def _look_again(camera):
    """A camera set, as a viewport or an animation makes for each picture."""
    camera.setLookAt(camera.getLookFrom(), camera.getLookAt(), camera.getVUp())


def run(s):
    kind = s["kind"]
    if kind == "frame":
        _look_again(s["pt"].scene.camera)
        s["pt"].render()
        return s["pt"].getFrameBuffer(s["dst"])
    if kind == "batch":
        for r, scene in zip(s["renderers"], s["scenes"]):
            r.set_camera(scene.camera.to_struct())
        s["batch"].render()
        s["batch"].synchronize()
        return [r.framebuffer(dst) for r, dst in zip(s["renderers"], s["dst"])]
    if kind == "rays":
        hits, visits = s["pt"].traceRays(s["rays"], with_visits=s["visits"])
        out = {k: hits[k] if hits[k].dtype == np.float32 else hits[k].view(np.int32) for k in hits.dtype.names}
        if visits is not None:
            out["visits"] = visits.view(np.int32)
        return out
    if kind == "infer":
        return s["cache"].infer(s["x"])
    if kind == "grads":
        grads, loss = s["cache"].gradients(s["x"], s["target"])
        return {"grads": grads, "loss": loss}
    if kind == "jpeg":
        return textures.read_jpeg(s["file"], flip_y=s["flip"])
    bvh = ornament.Bvh(s["scene"], builder=s["tree"])
    r = ornament.Renderer(bvh)
    r.close()
    return {"tlas": bvh.tlas_nodes.view(np.int32), "blas": bvh.blas_nodes.view(np.int32), "normals": bvh.normals,
            "uvs": bvh.uvs, "transforms": bvh.transforms, "materials": bvh.materials.view(np.int32)}


# ---- what a call cannot do without --------------------------------------------------------------

# triangles or spheres a ray may hit (instances counted), and bytes of scene data, rounded
PRIMS = {"small": 6e3, "spheres": 490, "instanced": 9e6, "large": 3e7, "room": 17}
SCENE_BYTES = {"small": 2e5, "spheres": 6e4, "instanced": 4e7, "large": 1.4e8, "room": 5e3}
BOX_FLOPS, HIT_FLOPS, SHADE_FLOPS = 18, 40, 150   # one slab test, one primitive test, one shaded vertex
MLP_MACS = 256 * 64 + 4 * 64 * 64 + 64 * 3


def _ray_flops(scene):
    """A ray has to be told from every primitive but the one it hits: two
    slab tests per halving of the scene and one primitive test."""
    return 2 * BOX_FLOPS * math.log2(PRIMS[scene]) + HIT_FLOPS


def work(case):
    kind = case["kind"]
    if kind == "frame":
        px = case["width"] * case["height"]
        samples = px * case["spp"] * max(1, case["streams"])
        rays = samples * 1.9   # rays per sample that the sphere and mesh fields average
        # per pixel the RNG state read and written, the accumulation and the framebuffer written, the latter read back
        return {"bytes": SCENE_BYTES[case["scene"]] + px * (8 + 16 + 32), "flops": rays * (_ray_flops(case["scene"]) + SHADE_FLOPS)}
    if kind == "batch":
        sizes = [(max(64, int(case["width"] * (1.0, 0.5, 0.2)[i % 3])), (1.0, 0.25, 4.0)[i % 3]) for i in range(case["count"])]
        px = sum(w * w * 9 // 16 for w, _ in sizes)
        samples = sum(w * w * 9 // 16 * max(1, int(case["spp"] * k)) for w, k in sizes)
        return {"bytes": case["count"] * case["tris"] * 64 + px * 56,
                "flops": samples * 1.5 * (_ray_flops("small") + SHADE_FLOPS)}
    if kind == "rays":
        return {"bytes": case["n"] * (24 + 32 + (4 if case["visits"] else 0)), "flops": case["n"] * _ray_flops(case["scene"])}
    if kind == "infer":
        return {"bytes": case["n"] * 52 + 135_168, "flops": case["n"] * 2 * MLP_MACS}
    if kind == "grads":
        return {"bytes": case["n"] * 52 + 2 * 135_168, "flops": case["n"] * 2 * (3 * MLP_MACS - 256 * 64)}
    if kind == "jpeg":
        px = case["width"] * case["height"]
        return {"bytes": px * 4.6, "flops": px * 3 * 32 + px * 10}
    tris = case["meshes"] * 20 * case["freq"] ** 2
    # vertices and indices read, two 64-byte nodes per triangle written on the host and again on the device
    return {"bytes": tris * (8 + 3 * 12 + 2 * 2 * 64), "flops": tris * 2 * BOX_FLOPS}


# ---- values in 64 bits --------------------------------------------------------------------------


def _forward64(weights, x):
    x = x.astype(np.float64)
    ang = np.pi * x[:, :, None] * 2.0 ** np.arange(12)
    enc = np.stack([np.sin(ang), np.cos(ang)], -1).reshape(len(x), 240)
    a = np.concatenate([enc, x, np.ones((len(x), 1)), np.zeros((len(x), 5))], 1)
    acts = []
    for i, w in enumerate(weights):
        acts.append(a)
        z = a @ w.astype(np.float64).T
        a = np.maximum(z, 0.0) if i < 5 else z
    return acts, a


def exact(case, seed):
    """The network's outputs, or its loss and gradients, in 64 bits.  Pictures,
    hits, texels and trees have none: a path's every decision hangs on its
    32-bit values, and the others are whole numbers."""
    if case["kind"] not in ("infer", "grads"):
        return None
    weights, x, target = _mlp_inputs(case, seed)
    acts, y = _forward64(weights, x)
    y = y[:, :3]
    if case["kind"] == "infer":
        return y
    has = target[:, :1] >= 0.0
    r = target.astype(np.float64)
    den = y * y + 0.01
    loss = float((np.where(has, (y - r) ** 2 / den, 0.0)).sum())
    dz = np.zeros((len(x), 16))
    dz[:, :3] = np.where(has, np.clip(2.0 * (y - r) / den, -1e4, 1e4), 0.0)
    grads = []
    for i in range(5, -1, -1):
        grads.append((dz.T @ acts[i]).ravel())
        if i:
            dz = (dz @ weights[i].astype(np.float64)) * (acts[i] > 0.0)
    return {"grads": np.concatenate(grads[::-1]), "loss": loss}


# ---- a JPEG file --------------------------------------------------------------------------------


def _zigzag():
    order = sorted(range(64), key=lambda i: (i // 8 + i % 8, i % 8 if (i // 8 + i % 8) % 2 == 0 else i // 8))
    return np.array(order)


def _code_lengths(symbols):
    """Code length of each symbol, most frequent first: a complete profile of
    2 to 11 bits for the first 46, 16 bits for the rest."""
    profile = [2] * 2 + [3] + [4] * 2 + [5] * 3 + [6] * 3 + [7] * 5 + [8] * 6 + [9] * 8 + [10] * 8 + [11] * 8
    return np.array((profile + [16] * len(symbols))[: len(symbols)])


def _codes(values, alphabet):
    """(table segment bytes, code of each symbol, length of each symbol)."""
    count = np.bincount(values, minlength=256)[:256]
    symbols = sorted(range(256), key=lambda v: -int(count[v]))
    symbols = [v for v in symbols if count[v] or v in alphabet]
    lengths = _code_lengths(symbols)
    code, length = np.zeros(256, np.int64), np.zeros(256, np.int64)
    c, last = 0, 0
    for v, n in zip(symbols, lengths):
        c <<= int(n) - last
        last = int(n)
        code[v], length[v] = c, n
        c += 1
    bits = [int((lengths == n).sum()) for n in range(1, 17)]
    return bytes(bits) + bytes(symbols), code, length


def _jpeg_file(width, height, seed):
    """A baseline 4:4:4 JPEG of a smooth picture with some grain and edges."""
    rs = np.random.default_rng(seed)
    w8, h8 = -(-width // 8) * 8, -(-height // 8) * 8
    y, x = np.mgrid[0:h8, 0:w8].astype(np.float32)
    planes = []
    for c in range(3):
        f = rs.uniform(0.004, 0.03, 4)
        p = 40 * np.sin(f[0] * x + 3 * np.sin(f[1] * y)) + 40 * np.cos(f[2] * y + f[3] * x)
        p += rs.normal(0, 4.0 if c == 0 else 1.0, p.shape).astype(np.float32)
        if c == 0:
            for _ in range(12):   # hard-edged rectangles
                x0, y0 = int(rs.integers(0, w8)), int(rs.integers(0, h8))
                p[y0:y0 + h8 // 6 + 1, x0:x0 + w8 // 8 + 1] += float(rs.uniform(-40, 40))
        planes.append(np.clip(p, -127, 127))
    u = np.arange(8)
    dct = 0.5 * np.cos((2 * u[None, :] + 1) * u[:, None] * np.pi / 16) * np.where(u == 0, math.sqrt(0.5), 1.0)[:, None]
    q = np.minimum(255, 6 + 3 * (u[:, None] + u[None, :])).reshape(64)
    zz = _zigzag()
    coef = []
    for p in planes:
        b = p.reshape(h8 // 8, 8, w8 // 8, 8).transpose(0, 2, 1, 3).astype(np.float32)
        f = np.matmul(np.matmul(dct.astype(np.float32), b), dct.T.astype(np.float32)).reshape(-1, 64)
        coef.append(np.rint(f / q)[:, zz].astype(np.int64))
    blocks = np.stack(coef, 1).reshape(-1, 64)                      # one block per component in each MCU
    dc = np.stack([np.diff(c[:, 0], prepend=0) for c in coef], 1).reshape(-1)
    size = lambda v: np.where(v == 0, 0, np.floor(np.log2(np.maximum(np.abs(v), 1))).astype(np.int64) + 1)  # noqa: E731
    extra = lambda v, n: np.where(v >= 0, v, v + (1 << n) - 1)  # noqa: E731
    n_blocks = len(blocks)
    bi, k = np.nonzero(blocks[:, 1:])
    k = k + 1
    v = blocks[bi, k]
    first = np.r_[True, bi[1:] != bi[:-1]] if len(bi) else np.zeros(0, bool)
    gap = k - np.where(first, 0, np.r_[0, k[:-1]][: len(k)]) - 1
    long_runs = gap // 16
    zrl = np.repeat(np.arange(len(bi)), long_runs)
    last = np.zeros(n_blocks, np.int64)
    np.maximum.at(last, bi, k)
    open_end = np.nonzero(last < 63)[0]
    key = np.concatenate([np.arange(n_blocks) * 256, bi * 256 + 2 * k + 1, bi[zrl] * 256 + 2 * k[zrl], open_end * 256 + 255])
    sd, sa = size(dc), size(v)
    ac_symbol = (gap % 16) * 16 + sa
    symbol = np.concatenate([sd, ac_symbol, np.full(len(zrl), 0xF0), np.zeros(len(open_end), np.int64)])
    dc_table, dc_code, dc_len = _codes(sd, range(12))
    ac_table, ac_code, ac_len = _codes(symbol[n_blocks:], (0x00, 0xF0))
    is_dc = np.arange(len(key)) < n_blocks
    code = np.where(is_dc, dc_code[symbol], ac_code[symbol])
    clen = np.where(is_dc, dc_len[symbol], ac_len[symbol])
    xbits = np.concatenate([extra(dc, sd), extra(v, sa), np.zeros(len(zrl) + len(open_end), np.int64)])
    xlen = np.concatenate([sd, sa, np.zeros(len(zrl) + len(open_end), np.int64)])
    order = np.argsort(key, kind="stable")
    word, n = ((code << xlen) | xbits)[order], (clen + xlen)[order]
    ends = np.cumsum(n)
    at = np.repeat(ends, n) - 1 - np.arange(int(ends[-1]))
    bit = (np.repeat(word, n) >> at) & 1
    data = np.packbits(np.r_[bit, np.ones(-len(bit) % 8, np.int64)].astype(np.uint8))
    data = np.insert(data, np.nonzero(data == 0xFF)[0] + 1, 0)      # byte stuffing

    def segment(marker, body):
        return bytes([0xFF, marker]) + (len(body) + 2).to_bytes(2, "big") + body

    head = b"\xff\xd8" + segment(0xE0, b"JFIF\0\1\1\0\0\1\0\1\0\0") + segment(0xDB, b"\0" + bytes(q[zz].tolist()))
    head += segment(0xC0, b"\x08" + height.to_bytes(2, "big") + width.to_bytes(2, "big") + b"\3" + b"".join(
        bytes([c, 0x11, 0]) for c in (1, 2, 3)))
    head += segment(0xC4, b"\x00" + dc_table) + segment(0xC4, b"\x10" + ac_table)
    return head + segment(0xDA, b"\3\1\0\2\0\3\0\0\x3f\0") + data.tobytes() + b"\xff\xd9"

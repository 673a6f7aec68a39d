"""The work a user of this framework has it do, as timed cases.

Every case goes through the public entry points (``GpuPipelineState`` and the
device-array primitives). Scenes follow ``cindergs_b200.scene.random_scene``
(normal means, log-uniform scales, uniform rotations, logit-normal opacities,
SH coefficients with a dominant DC term), drawn on the GPU from the seed;
cages and cameras are those of ``cindergs_b200.workloads``.

Kinds of case:

* ``viewer``   one frame call and the synchronous RGBA8 readback, as an
               interactive viewer with an orbiting camera makes it;
* ``views``    a step of one or more views into device images
               (``execute_views``), over a static scene, a spring-driven tet
               cage (optionally with strain splitting and the Mip filter) or
               a polygon cage bound exactly or through the learned field;
* ``infer``    the learned field evaluated for new points;
* ``train``    steps of the learned field's training;
* ``weights``  exact mean value coordinates of new points (training targets,
               bindings);
* ``sort``     the stable pair sort of the stage primitives.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cindergs_b200 import (Cage, CageScene, GaussianSceneSoa, GpuPipelineState, PolyCageMesh,
                           QuantizedGaussianSceneSoa, TetMesh, radix_sort_u32_pairs)
from cindergs_b200.camera import CameraUniforms, CompositorUniforms, orbit_camera
from cindergs_b200.workloads import spiral_views

DEV = "cuda:0"
FRAMES = 120  # frames per camera revolution
HID, FEATURES = 128, 64
CELLS = 5     # 5 x 5 x 5 cubes: 750 tets, 216 vertices


def listed():
    return [
        # a viewer's smallest frame: latency of the whole call, pixels on the host
        dict(name="viewer_20k_360p", kind="viewer", n=20_000, w=640, h=360, f16=False, deg=3,
             box=True),
        # a static scene at 720p, one view into a device image
        dict(name="static_100k_720p", kind="views", cage="none", n=100_000, w=1280, h=720,
             views=1, graph=False, f16=False, deg=3, tile=0, quant=False, box=True),
        # spring cage with strain splitting and the Mip filter, f16 SH, ragged size
        dict(name="split_300k_ragged", kind="views", cage="split", n=300_001, w=1283, h=717,
             views=1, graph=False, f16=True, deg=2, tile=0, quant=False, box=True),
        # the main workload: a spring-driven tet cage at 1080p
        dict(name="tet_1100k_1080p", kind="views", cage="tet", n=1_100_000, w=1920, h=1080,
             views=1, graph=False, f16=False, deg=3, tile=0, quant=False, box=True),
        # many views per step at mixed resolutions as a replayed graph, 32x16 tiles
        dict(name="views_2m_x12", kind="views", cage="tet", n=2_000_000, w=0, h=0, views=12,
             graph=True, f16=False, deg=3, tile=2, quant=False, box=False),
        # a quantized scene at 8K: 64-bit keys, hundreds of millions of tile entries
        dict(name="quant_1500k_8k", kind="views", cage="tet", n=1_500_000, w=7680, h=4320,
             views=1, graph=False, f16=True, deg=3, tile=0, quant=True, box=True),
        # polygon cage with exact stored bindings
        dict(name="mvc_exact_200k_1080p", kind="views", cage="mvc", n=200_000, w=1920, h=1080,
             views=1, graph=False, f16=False, deg=3, tile=0, quant=False, box=True),
        # polygon cage through the learned field, codes kept per Gaussian
        dict(name="mvc_learned_1m_1080p", kind="views", cage="learned", n=1_000_000, w=1920,
             h=1080, views=1, graph=False, f16=False, deg=3, tile=0, quant=False, box=True),
        # the learned field for points that have no codes
        dict(name="field_infer_250k", kind="infer", n=250_007, level=3),
        # training steps of the learned field
        dict(name="field_train_b4096", kind="train", n=65_536, batch=4096, steps=8, level=3),
        # exact weights of new points against the 642-vertex cage
        dict(name="mvc_weights_20k", kind="weights", n=20_011, level=3),
        # the pair sort on device arrays, 32-bit keys
        dict(name="sort_pairs_3m", kind="sort", n=3_000_001, bits=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the ranges of the listed ones."""
    kind = rng.choice(["viewer", "static", "tet", "tet", "split", "multi", "quant", "mvc",
                       "learned", "infer", "train", "weights", "sort"])
    w = _log(rng, 320, 1920)
    h = max(180, min(1080, int(w * rng.uniform(0.5, 0.75))))
    f16, deg, tile = rng.random() < 0.3, rng.choice([0, 1, 2, 3, 3]), rng.choice([0, 0, 1, 2])
    if kind == "viewer":
        return dict(kind="viewer", n=_log(rng, 5_000, 300_000), w=min(w, 1280), h=min(h, 720),
                    f16=f16, deg=deg, box=True)
    if kind in ("static", "tet", "split"):
        return dict(kind="views", cage="none" if kind == "static" else kind,
                    n=_log(rng, 10_000, 1_200_000), w=w, h=h, views=1, graph=False, f16=f16,
                    deg=deg, tile=tile, quant=False, box=True)
    if kind == "multi":
        return dict(kind="views", cage=rng.choice(["none", "tet"]), n=_log(rng, 20_000, 1_000_000),
                    w=0, h=0, views=rng.randint(2, 12), graph=rng.random() < 0.6, f16=f16, deg=3,
                    tile=rng.choice([0, 2]), quant=False, box=rng.random() < 0.5)
    if kind == "quant":
        return dict(kind="views", cage="tet", n=_log(rng, 100_000, 1_000_000),
                    w=rng.randint(5_000, 7_680), h=rng.randint(3_600, 4_320), views=1,
                    graph=False, f16=True, deg=rng.choice([1, 2, 3]), tile=0, quant=True, box=True)
    if kind == "mvc":
        return dict(kind="views", cage="mvc", n=_log(rng, 5_000, 150_000), w=w, h=h, views=1,
                    graph=False, f16=f16, deg=deg, tile=0, quant=False, box=True)
    if kind == "learned":
        return dict(kind="views", cage="learned", n=_log(rng, 10_000, 1_000_000), w=w, h=h,
                    views=1, graph=False, f16=f16, deg=deg, tile=0, quant=False, box=True)
    level = rng.choice([2, 3])
    if kind == "infer":
        return dict(kind="infer", n=_log(rng, 1_000, 400_000), level=level)
    if kind == "train":
        return dict(kind="train", n=_log(rng, 8_192, 65_536), batch=8 * _log(rng, 64, 512),
                    steps=rng.randint(4, 12), level=level)
    if kind == "weights":
        return dict(kind="weights", n=_log(rng, 500, 30_000), level=level)
    return dict(kind="sort", n=_log(rng, 1_000, 4_000_000), bits=rng.choice([16, 24, 32]))


# ---- inputs -------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _scene(c, g, ball=False):
    """random_scene's distribution, drawn on the GPU."""
    n = c["n"]
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV)  # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    pos = randn(n, 3)
    if ball:  # uniform in the unit ball, inside the polygon cage
        pos = pos / pos.norm(dim=1, keepdim=True).clamp_min(1e-9) * rand(n, 1) ** (1.0 / 3.0)
    elif c["box"]:
        pos = pos / pos.abs().max()
    scale = torch.exp(rand(n, 3) * 2.5 - 4.5).clamp_min(1e-4)
    q = randn(n, 4)
    q = q / q.norm(dim=1, keepdim=True).clamp_min(1e-9)
    w, x, y, z = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)],
                    1).reshape(n, 3, 3)
    M = R * scale[:, None, :]
    S = (M[:, :, None, :] * M[:, None, :, :]).sum(3)
    cov = torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 0, 2], S[:, 1, 1], S[:, 1, 2], S[:, 2, 2]], 1)
    opa = torch.sigmoid(randn(n))
    if c.get("quant"):
        bases = (c["deg"] + 1) ** 2
        words = (3 * bases + 1) // 2
        sh = randn(n, 2 * words) * 0.05
        sh[:, :3] *= 10.0
        sh[:, 3 * bases:] = 0.0
        return QuantizedGaussianSceneSoa(
            _host(pos), _host(cov.half().view(torch.int32)).view(np.uint32), _host(opa),
            _host(sh.half().view(torch.int32)).view(np.uint32), c["deg"])
    sh = randn(n, 48) * 0.05
    sh[:, :3] *= 10.0
    return GaussianSceneSoa(_host(pos), _host(cov), _host(opa),
                            _host(sh.half()) if c.get("f16") else _host(sh))


def _tet_cage(seed):
    """The spring-driven grid cage of ``workloads.tet_cage_orbit``."""
    mesh = TetMesh.create_grid_cage((CELLS,) * 3, (-1.1,) * 3, (1.1,) * 3)
    cage = Cage("grid", mesh)
    sim = cage.simulator
    sim.stiffness = np.float32(40.0)
    sim.damping = np.float32(np.exp(-4.0 / 60.0))
    sim.pinned = mesh.rest_vertices[:, 1] <= mesh.rest_vertices[:, 1].min()
    disp = np.random.default_rng(seed).normal(0.0, 0.05, mesh.rest_vertices.shape).astype(np.float32)
    disp[sim.pinned] = 0.0
    sim.current_positions = (mesh.rest_vertices + disp).astype(np.float32)
    return cage


def _poly_cage(level, seed):
    return PolyCageMesh.icosphere([0.0, 0.0, 0.0], 1.15, level).displace_sinusoids(0.1, 8, seed=seed)


def _moved(cage, frame, seed):
    """Cage vertices displaced by a smooth field moving with the frame."""
    rng = np.random.default_rng(seed + 5)
    k, ph = rng.normal(size=(3, 3)) * 2.0, rng.uniform(0, 6.28, 3)
    v = cage.rest_vertices.astype(np.float64)
    return (v + 0.05 * np.sin(v @ k.T + ph + 0.04 * frame)).astype(np.float32)


def _ball(n, g):
    p = torch.randn(n, 3, generator=g, device=DEV)
    p = p / p.norm(dim=1, keepdim=True).clamp_min(1e-9)
    return (p * torch.rand(n, 1, generator=g, device=DEV) ** (1.0 / 3.0)).contiguous()


def _offsets(V):
    """Parameter block: W1, b1, .., W5, b5, each padded to 8 floats."""
    sizes = [HID * FEATURES, HID, HID * HID, HID, HID * HID, HID, HID * HID, HID, V * HID, V]
    off = [0]
    for s in sizes:
        off.append(off[-1] + (s + 7) // 8 * 8)
    return sizes, off


def _params(V, seed):
    """A network of the trained one's scale: He-initialised hidden layers, a
    small output layer around equal weights."""
    sizes, off = _offsets(V)
    rng = np.random.default_rng(seed + 3)
    p = np.zeros(off[-1], np.float32)
    for k, fan in ((0, FEATURES), (2, HID), (4, HID), (6, HID)):
        p[off[k]:off[k] + sizes[k]] = rng.normal(0.0, math.sqrt(2.0 / fan), sizes[k])
    for k in (1, 3, 5, 7):
        p[off[k]:off[k] + sizes[k]] = rng.normal(0.0, 0.05, sizes[k])
    p[off[8]:off[8] + sizes[8]] = rng.normal(0.0, 1e-3, sizes[8])
    p[off[9]:off[9] + sizes[9]] = 1.0 / V
    return p


def _train_targets(V, n, g):
    """Positive weights that sum to one, the exact weights' range (mean 1/V)."""
    w = torch.rand(n, V, generator=g, device=DEV) ** 4
    return (w / w.sum(1, keepdim=True)).contiguous()


def _field_state(c, seed):
    cage = _poly_cage(c["level"], 0)
    p = GpuPipelineState(0)
    p.mvc_cage_upload(cage)
    p.mvc_field_create(seed=1)
    p.mvc_field_params(_params(cage.num_vertices, seed))
    return cage, p


def prepare(case, seed):
    c, g = dict(case), _gen(seed)
    kind = c["kind"]
    if kind == "viewer":
        scene = _scene(c, g)
        p = GpuPipelineState(0)
        p.upload_scene(scene)
        p.upload_cages(None)
        return dict(c=c, p=p, scene=scene, frame=seed % FRAMES)
    if kind == "views":
        poly = c["cage"] in ("mvc", "learned")
        scene = _scene(c, g, ball=poly)
        p = GpuPipelineState(0)
        p.upload_scene(scene)
        s = dict(c=c, p=p, scene=scene, frame=seed % FRAMES, cages=None, seed=seed)
        if c["cage"] in ("tet", "split"):
            s["cages"] = CageScene.auto_bind([_tet_cage(seed)], p, c["n"])
            p.upload_cages(s["cages"])
            p.springs_upload(s["cages"])
        else:
            p.upload_cages(None)
        if poly:
            s["poly"] = _poly_cage(3, 0)
            p.mvc_cage_upload(s["poly"])
            if c["cage"] == "mvc":
                p.mvc_bind()
            else:
                p.mvc_field_create(seed=1)
                p.mvc_field_params(_params(s["poly"].num_vertices, seed))
                p.mvc_bind_learned(1e6)
        if c["w"]:
            size = [CompositorUniforms(c["w"], c["h"])] * c["views"]
        else:  # mixed resolutions on a spiral: the same cameras every step
            s["cams"], s["comps"] = spiral_views(c["views"])
            size = s["comps"]
        s["images"] = p.view_images(size)
        return s
    if kind == "infer":
        cage, p = _field_state(c, seed)
        p.mvc_vertices_update(_moved(cage, 1, seed))
        return dict(c=c, p=p, pts=_ball(c["n"], g))
    if kind == "train":
        cage, p = _field_state(c, seed)
        return dict(c=c, p=p, pts=_ball(c["n"], g), tgt=_train_targets(cage.num_vertices, c["n"], g),
                    seed=seed + 1)
    if kind == "weights":
        p = GpuPipelineState(0)
        p.mvc_cage_upload(_poly_cage(c["level"], 0))
        return dict(c=c, p=p, pts=_ball(c["n"], g))
    stream = torch.cuda.Stream()
    p = GpuPipelineState(0, stream=stream.cuda_stream)
    hi = 1 << c["bits"]
    keys = torch.randint(0, hi, (c["n"],), generator=g, device=DEV).to(torch.int32)
    vals = torch.arange(c["n"], device=DEV, dtype=torch.int32)
    torch.cuda.synchronize()
    return dict(c=c, p=p, keys=keys, vals=vals, stream=stream)


# ---- passes -------------------------------------------------------------------

def _camera(c, frame):
    cam = orbit_camera(frame % FRAMES, FRAMES, 4.0, c["w"], c["h"], 60.0)
    comp = CompositorUniforms(c["w"], c["h"], (0.0, 0.0, 0.0, 1.0),
                              tuple(float(x) for x in cam.eye()), c["deg"])
    return cam, comp


def run(s):
    c, p = s["c"], s["p"]
    kind = c["kind"]
    if kind == "viewer":
        s["frame"] += 1
        cam, comp = _camera(c, s["frame"])
        p.execute_frame_gpu(s["scene"], None, cam, comp, stage_timings=False)
        return p.readback_framebuffer_rgba8(c["w"], c["h"])
    if kind == "views":
        s["frame"] += 1
        if s["cages"] is not None:
            p.springs_step(1.0 / 60.0)
        elif "poly" in s:
            p.mvc_vertices_update(_moved(s["poly"], s["frame"], s["seed"]))
        if c["w"]:
            cams, comps = zip(*[_camera(c, s["frame"] + 7 * v) for v in range(c["views"])])
        else:
            cams, comps = s["cams"], s["comps"]
        split = 1.3 if c["cage"] == "split" else 0.0
        p.execute_views(s["scene"], s["cages"], cams, comps, s["images"], use_graph=c["graph"],
                        strain_split_threshold=split, mip_filter_3d_var=0.001 if split else 0.0,
                        tile_shape=c["tile"])
        return s["images"]
    if kind == "infer":
        return list(p.mvc_field_infer(s["pts"]))
    if kind == "train":
        p.mvc_field_train(s["pts"], s["tgt"], steps=c["steps"], batch=c["batch"], lr=2e-3,
                          lam=0.05, seed=s["seed"])
        return p.mvc_field_params()
    if kind == "weights":
        return p.mvc_weights(s["pts"])
    with torch.cuda.stream(s["stream"]):
        k, v = s["keys"].clone(), s["vals"].clone()
        radix_sort_u32_pairs(p, k.data_ptr(), v.data_ptr(), c["n"], key_bits=c["bits"])
    return [k, v]


def _cage_size(level):
    return 10 * 4 ** level + 2, 20 * 4 ** level


def work(case):
    c = dict(case)
    kind, n = c["kind"], c["n"]
    if kind in ("viewer", "views"):
        sh = {0: 3, 1: 12, 2: 27, 3: 48}[c["deg"]] * (2 if c.get("f16") else 4)
        views = c.get("views", 1)
        px = c["w"] * c["h"] * views if c["w"] else sum(
            (230_400, 921_600, 2_073_600)[v % 3] for v in range(views))
        nbytes = n * (40 + sh) * views + 4 * px
        flops = n * 700.0 * views
        cage = c.get("cage", "none")
        if cage in ("tet", "split"):
            nbytes += 20 * n
        elif cage == "mvc":
            nbytes += n * 16 * _cage_size(3)[0]
            flops += n * 24.0 * _cage_size(3)[0]
        elif cage == "learned":
            nbytes += n * 1040
            flops += n * 2.0 * 4 * HID * 3
        return dict(bytes=nbytes, flops=flops)
    if kind == "sort":
        return dict(bytes=16 * n, flops=0)
    V, F = _cage_size(c["level"])
    net = FEATURES * HID + 3 * HID * HID
    if kind == "infer":
        return dict(bytes=n * 60 + 2 * (net + V * HID), flops=n * 8.0 * net)
    if kind == "train":
        rows = c["batch"] * c["steps"]
        return dict(bytes=rows * (4 * V + 12) + 4 * _offsets(V)[1][-1],
                    flops=6.0 * rows * (net + V * HID))
    return dict(bytes=n * (12 + 4 * V), flops=n * F * 150.0)


# ---- 64-bit values ------------------------------------------------------------

def _features64(x, enc):
    xh = (x - enc[:3]) * enc[3]
    f = [xh]
    for b in range(8):
        a = (2.0 ** b) * (math.pi / 2) * xh
        f.append(torch.stack([torch.sin(a), torch.cos(a)], 2).reshape(x.shape[0], 6))
    f = torch.cat(f, 1)
    return torch.cat([f, torch.zeros(x.shape[0], FEATURES - f.shape[1], device=x.device,
                                     dtype=x.dtype)], 1)


def _cage64(cage):
    v = torch.from_numpy(cage.rest_vertices.astype(np.float64)).to(DEV)
    lo, hi = v.min(0).values, v.max(0).values
    s = 0.5 * (hi - lo).max()
    enc = torch.cat([0.5 * (lo + hi), (1.0 / s)[None]])
    vb = torch.cat([torch.ones(1, v.shape[0], device=DEV, dtype=v.dtype), v.T])
    return v, enc, float(s), vb, torch.linalg.inv(vb @ vb.T)


def _split(p, V):
    sizes, off = _offsets(V)
    shapes = [(HID, FEATURES), (HID,), (HID, HID), (HID,), (HID, HID), (HID,), (HID, HID), (HID,),
              (V, HID), (V,)]
    return [p[off[k]:off[k] + sizes[k]].reshape(shapes[k]) for k in range(10)]


def _outputs64(x, q, enc):
    h = _features64(x, enc)
    for k in (0, 2, 4, 6):
        h = torch.nn.functional.silu(h @ q[k].T + q[k + 1])
    z = h @ q[8].T + q[9]
    return z + (1.0 - z.sum(1, keepdim=True)) / z.shape[1]


def _mix(z):
    """splitmix64's output function on uint64 arrays."""
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _train64(c, seed):
    cage = _poly_cage(c["level"], 0)
    V = cage.num_vertices
    g = _gen(seed)
    pts, tgt = _ball(c["n"], g).double(), _train_targets(V, c["n"], g).double()
    v, enc, s, vb, M = _cage64(cage)
    p = torch.from_numpy(_params(V, seed).astype(np.float64)).to(DEV)
    m, u = torch.zeros_like(p), torch.zeros_like(p)
    st = (seed + 1) ^ 0xD1B54A32D192ED03
    B, steps = c["batch"], c["steps"]
    for t in range(steps):
        bseed = (int(_mix(np.uint64(st))) & 0xFFFFFFFF) | 1  # _mix adds the increment itself
        st = (st + 0x9E3779B97F4A7C15) & 0xFFFFFFFFFFFFFFFF
        rows = (np.uint64(bseed) << np.uint64(32)) | np.arange(B, dtype=np.uint64)
        idx = torch.from_numpy(((_mix(rows) >> np.uint64(32)) % np.uint64(c["n"])).astype(np.int64)).to(DEV)
        x, w = pts[idx], tgt[idx]
        p.requires_grad_(True)
        w0 = _outputs64(x, _split(p, V), enc)
        r = w0 @ v - x
        one = torch.cat([torch.ones(B, 1, device=DEV, dtype=x.dtype), x], 1)
        e = w0 - (w0 @ vb.T - one) @ M @ vb - w
        loss = (e * e).sum() / B + 0.05 * (r * r).sum() / (3.0 * s * s) / B
        grad, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            lr = 2e-3 * (0.05 + 0.95 * 0.5 * (1.0 + math.cos(math.pi * t / steps)))
            m = 0.9 * m + 0.1 * grad
            u = 0.999 * u + 0.001 * grad * grad
            p = p.detach() - lr * (m / (1.0 - 0.9 ** (t + 1))) / (
                torch.sqrt(u / (1.0 - 0.999 ** (t + 1))) + 1e-8)
    return p.detach().cpu().numpy()


def _infer64(c, seed):
    cage = _poly_cage(c["level"], 0)
    v, enc, _, vb, M = _cage64(cage)
    cur = torch.from_numpy(_moved(cage, 1, seed).astype(np.float64)).to(DEV)
    q = [t.double() for t in _split(torch.from_numpy(_params(cage.num_vertices, seed)).to(DEV),
                                    cage.num_vertices)]
    pts, pos, F = _ball(c["n"], _gen(seed)), [], []
    for x in pts.double().split(32768):
        x = x.clone().requires_grad_(True)
        w0 = _outputs64(x, q, enc)
        one = torch.cat([torch.ones(x.shape[0], 1, device=DEV, dtype=x.dtype), x], 1)
        y = (w0 - (w0 @ vb.T - one) @ M @ vb) @ cur
        F.append(torch.stack([torch.autograd.grad(y[:, d].sum(), x, retain_graph=d < 2)[0]
                              for d in range(3)], 1))
        pos.append(y.detach())
    return [torch.cat(pos), torch.cat(F)]


def _weights64(c, seed):
    """Mean value coordinates of interior points (Ju, Schaefer and Warren 2005)."""
    cage = _poly_cage(c["level"], 0)
    v = torch.from_numpy(cage.rest_vertices.astype(np.float64)).to(DEV)
    tri = torch.from_numpy(cage.triangles.astype(np.int64)).to(DEV)
    out = []
    for x in _ball(c["n"], _gen(seed)).double().split(1024):
        d = v[None] - x[:, None]
        dist = d.norm(dim=2)
        u = d / dist[:, :, None]
        a, b, e = (u[:, tri[:, k]] for k in range(3))
        th = [2.0 * torch.asin((0.5 * (p - q).norm(dim=2)).clamp(max=1.0))
              for p, q in ((b, e), (e, a), (a, b))]
        hs = 0.5 * (th[0] + th[1] + th[2])
        det = (a * torch.linalg.cross(b, e)).sum(2)
        cs = [2.0 * torch.sin(hs) * torch.sin(hs - th[k]) /
              (torch.sin(th[(k + 1) % 3]) * torch.sin(th[(k + 2) % 3])) - 1.0 for k in range(3)]
        ss = [torch.sign(det) * torch.sqrt((1.0 - t * t).clamp(min=0.0)) for t in cs]
        w = torch.zeros_like(dist)
        for k in range(3):
            n1, n2 = (k + 1) % 3, (k + 2) % 3
            num = th[k] - cs[n1] * th[n2] - cs[n2] * th[n1]
            den = dist[:, tri[:, k]] * torch.sin(th[n1]) * ss[n2]
            m = torch.where(ss[n2].abs() > 1e-12, num / den, torch.zeros_like(num))
            w.index_add_(1, tri[:, k], m)
        out.append(w / w.sum(1, keepdim=True))
    return torch.cat(out)


def exact(case, seed):
    """Float outputs in 64 bits. Frames are bytes and sorts whole numbers."""
    c = dict(case)
    if c["kind"] == "infer":
        return _infer64(c, seed)
    if c["kind"] == "train":
        return _train64(c, seed)
    if c["kind"] == "weights":
        return _weights64(c, seed)
    return None

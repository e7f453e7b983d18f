"""Measured workloads of the GridNeRF renderer.

Each case is one call (or one short burst of calls) that a program built on this package makes
through its public entry points, on a seeded synthetic scene of the shapes in
``landmark_b200.scenes``.  The entry points:

* ``forward``     one chunk of rays through the model's ``forward``: rgb and depth of a few rays, or of one
                  render chunk;
* ``inferer``     a frame's rays through ``B200NerfDDPInfererImpl.renderer_fn``, the chunk loop of the offline
                  and online renderers (``render_batch_size`` rays per forward);
* ``frame``       a pose through ``NerfDDPRunner.run_batch``: uint8 image in host memory;
* ``pipe``        four poses submitted to ``PipeRunner``, then their images taken in order;
* ``host_rays``   ray buffers in pinned host memory through ``render_host``;
* ``points``      density and colour at explicit positions, what the owner of a block of a partitioned
                  scene computes for its peers.

Presets: ``exact`` (fp32 everywhere, the drop-in default), ``fast`` (fp16 tensor-core network, fp16 appearance
planes, pre-summed density, early termination), ``split`` (tensor-core network with activations as fp16 hi + lo,
for fields with large features), ``baked`` (``fast`` with the projected appearance features baked into a lattice).
Samplers: ``dense`` and ``hull`` (the online configurations).  Layouts: ``vm`` (three plane/line pairs) and
``multires`` (one direction at 1x/2x/4x, the layout of the city configurations).
"""
import math

import numpy as np
import torch

from landmark_b200 import scenes
from landmark_b200.engine import FrameRenderer, NerfDDPRunner
from landmark_b200.gridnerf import B200GridNeRF
from landmark_b200.inferer import PRESETS, B200NerfDDPInfererImpl
from landmark_b200.model_parallel import appearance_points, density_points
from landmark_b200.parallel import tile_pixel_ids
from landmark_b200.pipe_engine import PipeRunner, RunnerFrameBackend
from landmark_b200.rays import generate_rays

DEVICE = "cuda:0"


def _case(name, api, scene, width, height, samples, preset, rays=0, scale=1, chunk=0, sampler="dense", layout="vm",
          encode_app=False):
    """``rays`` = 0: every pixel of the image; otherwise that many rays of it.  ``scale`` divides the city grid."""
    c = {"api": api, "scene": scene, "scale": scale, "width": width, "height": height, "samples": samples, "preset": preset,
         "rays": rays, "chunk": chunk, "sampler": sampler, "layout": layout, "encode_app": encode_app}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a handful of rays: a colour/depth query under a cursor, a scattered subset of an evaluation image
        _case("rays_333_fast", "forward", "tiny", 100, 100, 128, "fast", rays=333),
        # one default render chunk (8192 rays) in the drop-in default precision
        _case("chunk_8192_exact", "forward", "city", 480, 270, 256, "exact", rays=8192, scale=8),
        # the small test image through the drop-in inferer, default precision and chunk size
        _case("tiny_100x100_exact", "inferer", "tiny", 100, 100, 128, "exact", chunk=8192),
        # an evaluation image through the same chunk loop with the fast preset
        _case("image_960x540_fast", "inferer", "city", 960, 540, 256, "fast", scale=4, chunk=8192),
        # preview frame of the online renderer
        _case("frame_480x270_fast", "frame", "city", 480, 270, 256, "fast", scale=8),
        # the benchmark frame of the online renderer
        _case("frame_1920x1080_fast", "frame", "city", 1920, 1080, 512, "fast"),
        # the same frame with every approximation off
        _case("frame_1920x1080_exact", "frame", "city", 1920, 1080, 512, "exact"),
        # online configuration: multi-resolution layout, hull sampler, an appearance code
        _case("frame_640x360_multires", "frame", "city", 640, 360, 128, "fast", scale=8, sampler="hull", layout="multires",
              encode_app=True),
        # odd-sized frame with the features baked into a lattice
        _case("frame_853x479_baked", "frame", "city", 853, 479, 384, "baked", scale=4),
        # a throughput run: several preview frames in flight
        _case("pipe_4x_640x360_fast", "pipe", "city", 640, 360, 256, "fast", scale=4),
        # a ragged number of host rays, hi + lo activations
        _case("host_150001_split", "host_rays", "city", 960, 540, 384, "split", rays=150001, scale=4, chunk=65536),
        # the owner of a block answers its peers' points
        _case("points_400003_fast", "points", "city", 960, 540, 256, "fast", rays=400003, scale=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    api = rng.choice(["forward", "forward", "inferer", "frame", "frame", "pipe", "host_rays", "points"])
    scene = "tiny" if api in ("forward", "inferer") and rng.random() < 0.4 else "city"
    scale = 1 if scene == "tiny" else rng.choice([2, 4, 8])
    preset = rng.choice(["exact", "exact", "fast", "fast", "fast", "split", "baked"])
    if api == "points":
        preset = "fast"  # block owners run the one-kernel appearance path
    layout = "multires" if preset not in ("baked",) and api != "points" and scene == "city" and rng.random() < 0.2 else "vm"
    if layout == "multires":
        scale = 8
    sampler = "hull" if layout == "multires" or (scene == "city" and rng.random() < 0.15) else "dense"
    samples = _log(rng, 64, 512 if sampler == "dense" else 256)
    tallest = {"frame": 720 if preset == "exact" else 1080, "pipe": 360 if preset == "exact" else 540}.get(api, 540)
    height = _log(rng, 40, tallest)
    width = height * 16 // 9 + rng.randint(-5, 5)
    rays = 0
    if api == "forward":
        rays = _log(rng, 64, 65536)
        height = max(height, 144)
        width = max(width, int(math.ceil(rays / height)) + 1)
    elif api in ("host_rays", "points"):
        rays = _log(rng, 4096, 400000)
        height = max(height, 144)
        width = max(width, int(math.ceil(rays / height)) + 1)
    chunk = {"inferer": rng.choice([4096, 8192, 16384]), "host_rays": 65536}.get(api, 0)
    return _case("", api, scene, width, height, samples, preset, rays=rays, scale=scale, chunk=chunk, sampler=sampler,
                 layout=layout, encode_app=rng.random() < 0.15 and preset != "exact" and api not in ("points",))


# ---- scene, model, camera -----------------------------------------------------------------------------------------
def _spec(case):
    if case["scene"] == "tiny":
        spec = scenes.tiny_spec(case["height"], case["width"], case["samples"])
    else:
        spec = scenes.city_spec(case["height"], case["width"], case["samples"], case["scale"])
    spec = spec.lit()
    spec.encode_app = case["encode_app"]
    return spec


def _checkpoint(case, spec, seed):
    if case["layout"] != "multires":
        return scenes.make_checkpoint(spec, seed=seed + 1, mask_seed=seed % (1 << 31), device=DEVICE)
    ckpt = scenes.make_checkpoint(spec, seed=seed + 1, mask_seed=seed % (1 << 31), device=DEVICE)
    g = torch.Generator(device=DEVICE).manual_seed(seed + 2)
    gx, gy, gz = spec.grid
    sd = {k: v for k, v in ckpt["state_dict"].items() if "plane" not in k and "line" not in k}
    for j, r in enumerate((1, 2, 4)):
        for kind, comps in (("density", spec.density_n_comp[0]), ("app", spec.app_n_comp[0])):
            sd[f"{kind}_plane.{j}"] = 0.1 * torch.randn((1, comps, gy * r, gx * r), generator=g, device=DEVICE)
            sd[f"{kind}_line.{j}"] = 0.1 * torch.randn((1, comps, gz * r, 1), generator=g, device=DEVICE)
    ckpt["state_dict"] = sd
    return ckpt


def _args(case, spec):
    args = scenes.model_args(spec, DEVICE)
    if case["layout"] == "multires":
        args.ndims, args.resMode = 1, [1, 2, 4]
    if case["sampler"] == "hull":
        args.sampling_opt, args.n_importance = 1, case["samples"]
    if case["chunk"]:
        args.render_batch_size = case["chunk"]
    return args


def _options(case):
    if case["preset"] == "split":
        opts = {"mlp_mode": 1, "ert_transmittance": 2e-5, "density_lattice": True}
    elif case["preset"] == "baked":
        opts = dict(PRESETS["fast"], appearance_lattice=True)
    else:
        opts = dict(PRESETS[case["preset"]])
    if case["layout"] == "multires":
        opts["density_lattice"] = False  # a pre-summed lattice needs one grid
    return opts


def _poses(case, spec, volume, seed, n):
    """Views of a viewer that moves: around the scene (tiny) or above the roofs, looking 30 degrees down (city)."""
    rng = np.random.RandomState((seed * 7919 + 13) % (1 << 32))
    out = []
    for _ in range(n):
        if case["scene"] == "tiny":
            el, az, r = math.radians(rng.uniform(15, 45)), rng.uniform(0, 2 * math.pi), 2.0
            eye = (r * math.cos(el) * math.cos(az), r * math.cos(el) * math.sin(az), r * math.sin(el))
            out.append(scenes.look_at(eye, (0.0, 0.0, 0.0)))
        else:
            d, h, w = volume.shape
            x, y = rng.uniform(-2.0, 2.0, size=2)
            col = volume[:, int((y / 16 + 0.5) * (h - 1)), int((x / 16 + 0.5) * (w - 1))].nonzero()
            top = spec.aabb[0][2] + (spec.aabb[1][2] - spec.aabb[0][2]) * ((int(col.max()) + 1) / d if col.numel() else 0.0)
            out.append(scenes.pitched_pose((x, y, top + 0.5), rng.uniform(0.0, 360.0), -30.0))
    return out


class _Context:
    def __init__(self, args, checkpoint):
        self.args_nerf, self.checkpoint, self.model_path = args, checkpoint, None


def prepare(case, seed):
    spec = _spec(case)
    ckpt = _checkpoint(case, spec, seed)
    args = _args(case, spec)
    volume = torch.from_numpy(np.unpackbits(ckpt["alphaMask.mask"])[: int(np.prod(ckpt["alphaMask.shape"]))]
                              .reshape(ckpt["alphaMask.shape"]))
    state = {"api": case["api"], "samples": case["samples"], "code": 7 if case["encode_app"] else None}
    h, w = case["height"], case["width"]
    poses = _poses(case, spec, volume, seed, 4)
    if case["api"] == "inferer":
        impl = B200NerfDDPInfererImpl(_Context(args, ckpt), **dict(_options(case), preset="exact"))
        impl.load_model(h, w)
        state["impl"] = impl
        model = impl.model
    else:
        kwargs = dict(ckpt["kwargs"])
        kwargs.update({"device": DEVICE, "args": args, "is_train": False})
        model = B200GridNeRF(**kwargs, **_options(case))
        model.load(ckpt)
    if state["code"] is not None:
        model.set_app_code(state["code"])
    state["model"] = model
    if case["api"] in ("frame", "pipe"):
        runner = NerfDDPRunner(FrameRenderer(model, n_samples=case["samples"]), h, w, spec.focal)
        state["runner"] = PipeRunner(RunnerFrameBackend(runner), depth=4) if case["api"] == "pipe" else runner
        state["poses"] = poses
        return state
    if case["api"] == "inferer":  # an image's rays in row order
        state["rays"] = generate_rays(poses[0], h, w, spec.focal, device=DEVICE)
        return state
    # rays in tile order, as a rank of a renderer holds them
    ids = torch.from_numpy(tile_pixel_ids(h, w, 0, 1)).to(DEVICE)
    rays = generate_rays(poses[0], h, w, spec.focal, device=DEVICE, pixel_ids=ids)
    n = case["rays"] or rays.shape[0]
    if case["api"] == "points":
        # samples of neighbouring rays at equal ranks, near the surfaces the camera sees
        t = torch.linspace(0.3, 4.0, 8, device=DEVICE)
        per = -(-n // t.numel())
        r = rays[torch.arange(per, device=DEVICE) % rays.shape[0]]
        pts = (r[None, :, :3] + t[:, None, None] * r[None, :, 3:]).reshape(-1, 3)[:n]
        state["xyz"] = model.normalize_coord(pts).clamp(-1.0, 1.0).contiguous()
        state["view"] = r[None, :, 3:].expand(t.numel(), -1, -1).reshape(-1, 3)[:n].contiguous()
        return state
    first = (rays.shape[0] - n) // 2
    rays = rays[first:first + n].contiguous()
    if case["api"] == "host_rays":
        state["rays"] = rays.cpu().pin_memory()
        state["rgb"] = torch.empty((n, 3)).pin_memory()
        state["depth"] = torch.empty((n,)).pin_memory()
        state["chunk"] = case["chunk"]
    else:
        state["rays"] = rays
    return state


def run(state):
    api, s = state["api"], state["samples"]
    if api == "forward":
        out, _ = state["model"](state["rays"], app_code=state["code"], white_bg=True, is_train=False, N_samples=s)
        return [out["rgb_map"], out["depth_map"]]
    if api == "inferer":
        return state["impl"].renderer_fn(state["rays"], N_samples=s, white_bg=True, app_code=state["code"])
    if api == "frame":
        return state["runner"].run_batch(state["poses"][0])
    if api == "pipe":
        for pose in state["poses"]:
            state["runner"].run_batch(pose)
        return [state["runner"].get_result() for _ in state["poses"]]
    if api == "host_rays":
        rgb, depth = state["model"].render_host(state["rays"], s, True, chunk=state["chunk"], rgb_out=state["rgb"],
                                                depth_out=state["depth"])
        return [rgb, depth]
    return [density_points(state["model"], state["xyz"]), appearance_points(state["model"], state["xyz"], state["view"])]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    """Bytes: the rays (or poses' images) in and out, and every field value once, at most as often as samples touch it.
    Flops: interpolation and network of the samples that reach them (mean counts per ray of these scenes)."""
    n = case["rays"] or case["width"] * case["height"]
    frames = 4 if case["api"] == "pipe" else 1
    s = case["samples"]
    if case["api"] == "points":
        den, app = float(n), float(n)
    else:
        # optical depth of one step in an occupied cell: density ln 2, distance scale 25; a sample is coloured while its
        # weight exceeds 1e-3, and a terminating ray stops at a transmittance of 2e-5; a third of the samples is occupied
        step = {"tiny": 0.0079, "city": 0.0039 * case["scale"]}[case["scene"]] if case["sampler"] == "dense" else 1.2 / s
        tau = 17.3 * step
        app = min(0.3 * s, math.log(1000.0 * (1.0 - math.exp(-tau))) / tau) * n
        den = (0.3 * s if case["preset"] == "exact" else min(0.3 * s, math.log(5e4) / tau)) * n
    den, app = den * frames, app * frames
    half = case["preset"] in ("fast", "baked")
    spec = _spec(case)
    gx, gy, gz = spec.grid
    texels = 21 * gx * gy if case["layout"] == "multires" else gx * gy + gx * gz + gy * gz
    if case["preset"] in ("fast", "split", "baked") and case["layout"] == "vm":
        den_field, den_tap = 4.0 * gx * gy * gz, 32.0
    else:
        den_field, den_tap = 64.0 * texels, 18 * 64.0
    if case["preset"] == "baked":
        app_field, app_tap = 64.0 * gx * gy * gz, 8 * 64.0
    else:
        app_field, app_tap = (96.0 if half else 192.0) * texels, 18 * (96.0 if half else 192.0)
    # one of a hundred texel reads is a new texel: neighbouring rays see the same texels
    field = min(den_field, 0.01 * den * den_tap) + min(app_field, 0.01 * app * app_tap)
    if case["api"] in ("frame", "pipe"):
        io = 4.0 * n * frames
    else:
        io = n * (24.0 + 16.0)
    return {"bytes": io + field + 4e5, "flops": app * 79712.0 + den * 700.0}


def tolerance(case):
    exact = case["preset"] == "exact"
    if case["api"] in ("frame", "pipe"):
        # images are truncated to bytes: a colour within rounding distance of a step may land on either side of it
        return {"rel": 2e-3, "max": 0.05, "differ": 1e-3 if exact else 5e-3}
    # `max`: a weight within rounding distance of the appearance threshold (1e-3) enters or leaves the colour sum
    if exact:
        return {"rel": 1e-5, "max": 5e-3}
    return {"rel": 2e-4, "max": 5e-3}

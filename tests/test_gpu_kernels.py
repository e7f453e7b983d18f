"""GPU tests of single kernels at the sizes where their work split has its edges: partial tiles and words, the
smallest and largest chunk a rule picks a form for.  References: the CPU oracle, or the same pixels computed another way."""
import ctypes as C

import numpy as np
import pytest
import torch

from landmark_b200 import scenes
from landmark_b200._lib import EXPIRE_ANY, EXPIRE_NETWORK, EXPIRE_PROJECTION
from oracle import sampling_numpy as snp
from tests._util import cuda_model, oracle_field, tiny_rays, valid_bits_from_words

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,samples,thres,mask", [
    (1, 1, 0.0, True), (3, 7, 0.0, True), (5, 32, 0.0, True), (33, 33, 0.0, True), (31, 100, 0.5, True), (130, 257, 0.0, True),
    (7, 1061, 0.0, True), (64, 96, 0.0, False), (6000, 64, 0.0, True), (160001, 40, 0.0, True)])
def test_sampler_words_at_edges(n, samples, thres, mask):
    """Words, counts and entry distances are equal bit for bit to the restatement that tests every sample: partial last
    words and runs, one ray per warp up to 32, more than 32 words per ray, both thresholds, no mask."""
    spec = scenes.tiny_spec().lit()
    spec.alpha_filter_thres = thres
    field, ckpt = oracle_field(spec)
    if not mask:
        ckpt = {k: v for k, v in ckpt.items() if not k.startswith("alphaMask")}
    model = cuda_model(spec, ckpt)
    g = torch.Generator().manual_seed(n + samples)
    o = torch.rand((n, 3), generator=g) * 2.4 - 1.2
    d = torch.randn((n, 3), generator=g)
    d[::4, 2] = 0.0
    o[::3] = (o[::3] * 16).round() / 16  # on lattice planes
    rays = torch.cat([o, d], 1).contiguous()
    got = model.run_stages(rays.cuda(), samples, True, upto="sample")
    volume = field.alpha_volume[0, 0].numpy() if mask else None
    valid, t_min = snp.valid_mask(rays.numpy(), field.aabb.numpy(), field.near, field.far, field.step_size.item(), samples,
                                  volume, field.alpha_aabb.numpy() if mask else None, thres)
    assert np.array_equal(valid_bits_from_words(got["mask_words"], samples), valid)
    assert np.array_equal(got["t_min"].cpu().numpy(), t_min)
    assert np.array_equal(got["counts"].cpu().numpy(), valid.sum(1))


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("n,samples,ert", [(1, 3, 0.0), (5, 128, 0.0), (37, 33, 0.0), (3071, 128, 0.0), (3073, 128, 0.0), (6150, 97, 0.0),
                                           (12290, 64, 0.0), (98400, 40, 0.0), (3075, 128, 0.3), (333, 128, 0.3)])
def test_march_forms_give_the_stagewise_bits(n, samples, ert, lattice):
    """Every number of lanes per ray (rule edges, a last group with one ray, one-sample rays): the pixels of forward equal
    the stage-wise pixels (one thread per ray, scanned offsets) bit for bit; with termination they equal the scanned form
    of the same kernel, which a capacity below the worst case selects."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec, density_lattice=lattice, ert_transmittance=ert)
    model.app_capacity_per_ray = 64
    rays = tiny_rays(spec).cuda()
    rays = rays.repeat((n + rays.shape[0] - 1) // rays.shape[0], 1)[:n].contiguous()
    out, _ = model(rays, N_samples=samples)
    got = model.last_status.copy()
    if ert == 0.0:
        ref = model.run_stages(rays, samples, True)
        assert got[2] == ref["num_valid"] and got[3] == ref["num_app"] and got[5] == ref["num_valid"]
    else:
        model.valid_capacity_per_ray = samples - 1
        ref, _ = model(rays, N_samples=samples)
        assert np.array_equal(got, model.last_status) and got[5] < got[2]
    assert torch.equal(out["rgb_map"], ref["rgb_map"]) and torch.equal(out["depth_map"], ref["depth_map"])


def test_appearance_list_overflow_is_reported():
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    rays = tiny_rays(spec).cuda()
    model.app_capacity_per_ray = 1
    for n in (200, 4000, 10000):
        with pytest.raises(RuntimeError, match="appearance-sample list overflow"):
            model(rays[5000 - n // 2:5000 + n // 2].contiguous(), N_samples=spec.n_samples)


def _network_fp64(sd, feats, view):
    """MLPRender_Fea in fp64, and a bound on the error of an fp32 evaluation: every layer's sums may be off by
    16 x 2^-24 of the sum of magnitudes (rounding of operands, encodings and bias, and ten accumulation steps at full
    size), propagated through the layers; sigmoid has slope 1/4 at most and one rounding of its own."""
    def pe(x):
        p = (x[..., None] * torch.tensor([1.0, 2.0], dtype=torch.float64, device=x.device)).reshape(x.shape[0], -1)
        return torch.cat([p.sin(), p.cos()], -1)

    gamma = 16 * 2.0 ** -24
    x = torch.cat([feats, view, pe(feats), pe(view)], -1)
    err = torch.zeros_like(x)
    for i in (0, 2, 4):
        w, b = sd[f"renderModule.mlp.{i}.weight"], sd[f"renderModule.mlp.{i}.bias"]
        err = err @ w.abs().T + gamma * (x.abs() @ w.abs().T + b.abs())
        x = x @ w.T + b
        if i < 4:
            x = torch.relu(x)
    return torch.sigmoid(x), 0.25 * err + 2.0 ** -24


@pytest.mark.parametrize("n,scale", [(1, 0.02), (127, 0.02), (128, 1.0), (129, 0.02), (148 * 128 + 1, 5.0), (3 * 148 * 128 + 77, 0.3)])
def test_fp32_network_on_tensor_cores(n, scale):
    """The fp32 network as sums of bf16 terms, from given features: inside the error bound of an fp32 evaluation against
    fp64 for partial tiles, one to four tiles per CTA, features from 0.02 to 5 (times a normal variable)."""
    from landmark_b200.model_parallel import mlp_features

    spec = scenes.tiny_spec(grid=32).lit()
    ckpt = scenes.make_checkpoint(spec)
    g = torch.Generator().manual_seed(n)
    ckpt["state_dict"]["renderModule.mlp.4.bias"] = torch.randn(3, generator=g)
    model = cuda_model(spec, ckpt)
    feats = (torch.randn((n, 27), generator=g) * scale).cuda()
    view = torch.randn((n, 3), generator=g).cuda()
    rgb = mlp_features(model, feats, view)
    ref, bound = _network_fp64({k: v.cuda().double() for k, v in ckpt["state_dict"].items()}, feats.double(), view.double())
    worst = ((rgb.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, f"error is {worst:.2f} of the bound"


def test_fp32_network_bits_do_not_depend_on_the_order_of_samples():
    """A few features beyond the range of the short sine among ordinary ones: every sample has the same bits in any order."""
    from landmark_b200.model_parallel import mlp_features

    spec = scenes.tiny_spec(grid=32).lit()
    model = cuda_model(spec)
    g = torch.Generator().manual_seed(1)
    feats, view = torch.randn((4097, 27), generator=g), torch.randn((4097, 3), generator=g)
    feats[::97, 3], feats[50::131, 26], view[7::500, 1] = 700.0, -1e6, 501.0
    order = torch.randperm(feats.shape[0], generator=g)
    rgb = mlp_features(model, feats.cuda(), view.cuda())
    assert torch.equal(rgb[order.cuda()], mlp_features(model, feats[order].cuda(), view[order].cuda()))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kernel", [EXPIRE_ANY, EXPIRE_PROJECTION, EXPIRE_NETWORK])
def test_fp32_network_wait_expires_and_the_context_survives(kernel, mode):
    """The projection and the network each report a wait that runs out (both write the chunk's one status block, so each is
    made to run out alone)."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec, mlp_mode=mode)
    rays = tiny_rays(spec).cuda()[4000:6000].contiguous()
    good, _ = model(rays, N_samples=spec.n_samples)
    model.debug_wait(expire=kernel, wait_limit=2000)
    with pytest.raises(RuntimeError, match="bounded device-side wait expired"):
        model(rays, N_samples=spec.n_samples)
    model.debug_wait()
    again, _ = model(rays, N_samples=spec.n_samples)
    assert torch.equal(good["rgb_map"], again["rgb_map"])


@pytest.mark.parametrize("mode", [0, 1])
def test_waits_that_run_out_at_once_leave_no_copy_behind(mode):
    """One poll per wait: roles of the split kernels give up while the copies of the weights are still on their way into
    shared memory.  The kernels see them out before they leave, so that the launches behind them read what they loaded."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec, mlp_mode=mode)
    rays = tiny_rays(spec).cuda()
    good, _ = model(rays, N_samples=spec.n_samples)
    model.check_status_every_call = False
    for _ in range(5):
        model.debug_wait(wait_limit=1)
        model(rays, N_samples=spec.n_samples)
        model.debug_wait()
        again, _ = model(rays, N_samples=spec.n_samples)
        assert torch.equal(good["rgb_map"], again["rgb_map"])


def test_inferer_chunks_fit_the_sample_ids():
    """65536 rays of 40000 samples do not fit the 32-bit ids of a chunk, 8192 do: the drop-in loop takes what fits."""
    from types import SimpleNamespace

    from landmark_b200.inferer import B200NerfDDPInfererImpl

    spec = scenes.tiny_spec(grid=32).lit()
    args = scenes.model_args(spec, "cuda:0")
    args.render_batch_size = 64
    impl = B200NerfDDPInfererImpl(SimpleNamespace(args_nerf=args, checkpoint=scenes.make_checkpoint(spec), model_path=None))
    impl.load_model(spec.height, spec.width)
    impl.model.app_capacity_per_ray = impl.model.valid_capacity_per_ray = 64
    rays = torch.zeros((65536, 6), device="cuda:0")
    rays[:, 2], rays[:, 5] = 50.0, 1.0  # above the scene, looking away: no valid sample
    assert torch.equal(impl.renderer_fn(rays, N_samples=40000), torch.ones_like(rays[:, :3]))


def test_frames_of_one_renderer_in_changing_chunks_and_images():
    """The frame call keeps its buffers per image and chunk count; images it cannot write as plain bytes, and renderers
    with stages of their own, take the stage-wise path.  All give the same bytes."""
    from landmark_b200.engine import FrameRenderer, NerfDDPRunner

    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    renderer = FrameRenderer(model, spec.n_samples, chunk=4096)
    runner = NerfDDPRunner(renderer, spec.height, spec.width, focal=spec.focal)
    pose = scenes.make_pose(spec)
    first = runner.run_batch(pose).copy()
    renderer.chunk = 500  # more status blocks than the ring had
    assert np.array_equal(first, runner.run_batch(pose))
    wide = torch.zeros((spec.height, spec.width, 8), dtype=torch.uint8).pin_memory()
    runner.enqueue(pose, wide[..., :4]).synchronize()
    assert np.array_equal(first, wide[..., :4].numpy()) and not wide[..., 4:].any()
    with pytest.raises(RuntimeError):
        runner.enqueue(pose, torch.zeros((spec.height, spec.width - 1, 4), dtype=torch.uint8).pin_memory())

    class Dark(FrameRenderer):
        def to_rgba8(self, image, out):
            super().to_rgba8(image * 0.0, out)

    dark = NerfDDPRunner(Dark(model, spec.n_samples), spec.height, spec.width, focal=spec.focal).run_batch(pose)
    assert not dark[..., :3].any() and (dark[..., 3] == 255).all()


@pytest.mark.parametrize("n,samples,thres,mask", [
    (1, 1, 0.0, True), (5, 33, 0.0, True), (130, 97, 0.5, True), (64, 128, 0.0, False), (6000, 64, 0.0, True), (3001, 1061, 0.0, True)])
def test_hull_sampler_words_at_edges(n, samples, thres, mask):
    """The hull sampler decides runs of samples from their ends too: words equal bit for bit to testing every sample, rays
    that look up, (almost) along the ground plane (far up to infinity, or 0 / 0 on it) and from below it among them."""
    from landmark_b200.gridnerf import B200GridNeRF

    spec = scenes.tiny_spec().lit()
    spec.alpha_filter_thres = thres
    field, ckpt = oracle_field(spec)
    if not mask:
        ckpt = {k: v for k, v in ckpt.items() if not k.startswith("alphaMask")}
    args = scenes.model_args(spec, "cuda:0")
    args.sampling_opt, args.n_importance = 1, samples
    kw = dict(ckpt["kwargs"])
    kw.update({"device": "cuda:0", "args": args, "is_train": False})
    model = B200GridNeRF(**kw)
    model.load(ckpt)
    g = torch.Generator().manual_seed(n + samples)
    o = torch.rand((n, 3), generator=g) * 3.0 - 1.5
    d = torch.randn((n, 3), generator=g)
    o[::3] = (o[::3] * 16).round() / 16
    d[1::5, 2] = -1e-38
    d[2::7, 2] = -0.0
    o[2::14, 2] = float(field.aabb[0, 2])
    rays = torch.cat([o, d], 1).contiguous()
    got = model.run_stages(rays.cuda(), samples, True, upto="sample")
    a = field.aabb.numpy()
    u = torch.linspace(0.0, 1.0, steps=samples)
    near_term, u = (field.near * (1.0 - u)).numpy(), u.numpy()
    with np.errstate(all="ignore"):
        far = -((o[:, 2].numpy() - a[0, 2]) / d[:, 2].numpy())
        far = np.where(d[:, 2].numpy() >= 0, np.float32(field.far), far)
        z = near_term[None] + far[:, None] * u[None]
        pts = o.numpy()[:, None] + d.numpy()[:, None] * z[:, :, None]
        valid = snp.in_box(pts, a)
        if mask:
            m = field.alpha_aabb.numpy()
            inv = (np.float32(1.0) / (m[1] - m[0])) * np.float32(2)
            q = (pts[valid] - m[0]) * inv - np.float32(1)
            finite = np.isfinite(q).all(1)
            alpha = np.zeros(len(q), np.float32)
            alpha[finite] = snp.trilinear_zero_pad(field.alpha_volume[0, 0].numpy(), q[finite])
            at = np.nonzero(valid)
            keep = alpha > np.float32(thres)
            valid[at[0][~keep], at[1][~keep]] = False
    assert z.dtype == pts.dtype == np.float32
    assert np.array_equal(valid_bits_from_words(got["mask_words"], samples), valid)
    assert np.array_equal(got["counts"].cpu().numpy(), valid.sum(1))


@pytest.mark.parametrize("options", [{}, {"mlp_mode": 1}, {"mlp_mode": 2, "app_plane_fp16": True, "density_lattice": True, "ert_transmittance": 2e-5}])
def test_chained_launches_keep_the_order_of_calls(options):
    """Chunks of changing size queued back to back into one workspace, the kernels of each chained, between copies and
    plain kernels of the caller: the pixels of every call equal those of the same call waited for by itself."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec, **options)
    rays = tiny_rays(spec).cuda()
    sizes = [1, 333, 9000, 40, 3100, 7000, 128, 2000] * 3
    starts = [(977 * i) % (rays.shape[0] - n + 1) for i, n in enumerate(sizes)]
    want = []
    for a, n in zip(starts, sizes):
        want.append(model(rays[a:a + n].contiguous(), N_samples=spec.n_samples)[0]["rgb_map"].clone())
        torch.cuda.synchronize()
    model.check_status_every_call = False
    staged = torch.empty_like(rays)
    got = []
    for a, n in zip(starts, sizes):
        staged[:n].copy_(rays[a:a + n])  # (into the buffer the call before still reads)
        got.append(model(staged[:n], N_samples=spec.n_samples)[0]["rgb_map"] * 1.0)
    for g, w in zip(got, want):
        assert torch.equal(g, w)


def _pairs_model(ndims, res_mode, channels, mode, **extra):
    """A model with any layout of plane/line pairs, on a grid whose taps are exact for positions of 1/256."""
    from landmark_b200.gridnerf import B200GridNeRF

    spec = scenes.tiny_spec(grid=17).lit()
    spec.app_n_comp = (channels,) * 3
    g = torch.Generator().manual_seed(100 * ndims + len(res_mode))
    sd = {k: v for k, v in scenes.make_state_dict(spec).items() if k.startswith("renderModule")}
    for i in range(ndims):
        m0, m1 = scenes.MAT_MODE[i]
        for j, r in enumerate(res_mode):
            size = [17 * r] * 3
            for kind, c in (("density", 16), ("app", channels)):
                sd[f"{kind}_plane.{i * len(res_mode) + j}"] = 0.1 * torch.randn((1, c, size[m1], size[m0]), generator=g)
                sd[f"{kind}_line.{i * len(res_mode) + j}"] = 0.1 * torch.randn((1, c, size[scenes.VEC_MODE[i]], 1), generator=g)
    k = ndims * len(res_mode) * channels
    sd["basis_mat.weight"] = (torch.rand((27, k), generator=g) * 2 - 1) / k ** 0.5
    ckpt = scenes.make_checkpoint(spec)
    ckpt["state_dict"] = sd
    args = scenes.model_args(spec, "cuda:0")
    args.ndims, args.resMode = ndims, list(res_mode)
    kw = dict(ckpt["kwargs"])
    kw.update({"device": "cuda:0", "args": args, "is_train": False})
    model = B200GridNeRF(**kw, mlp_mode=mode, **extra)
    model.load(ckpt)
    return model, sd


def _features_fp64(sd, ndims, n_res, xyz, magnitudes=False):
    """compute_appfeature in fp64; ``magnitudes``: the sums of the terms' magnitudes instead."""
    parts = []
    f = torch.abs if magnitudes else (lambda t: t)
    for i in range(ndims * n_res):
        d = i // n_res
        uv = xyz[:, list(scenes.MAT_MODE[d])].double().view(1, -1, 1, 2)
        line = xyz[:, scenes.VEC_MODE[d]].double()
        line = torch.stack([torch.zeros_like(line), line], -1).view(1, -1, 1, 2)
        p = torch.nn.functional.grid_sample(f(sd[f"app_plane.{i}"].cuda().double()), uv, align_corners=True)
        l = torch.nn.functional.grid_sample(f(sd[f"app_line.{i}"].cuda().double()), line, align_corners=True)
        parts.append((p * l)[0, :, :, 0].T)
    w = f(sd["basis_mat.weight"].cuda().double())
    return torch.cat(parts, 1) @ w.T, w


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("ndims,res_mode,channels", [
    (1, (1,), 48), (2, (1,), 48), (3, (1,), 48), (3, (1,), 16), (3, (1,), 24), (1, (1, 2, 4), 48), (2, (1, 2), 48), (2, (1, 2), 32),
    (1, (1, 2, 1, 2, 1), 48), (1, (1, 2, 1, 2, 1), 16), (3, (1, 2), 48), (3, (1, 2), 16), (1, (1, 2, 1, 2, 1, 2, 1), 32),
    (2, (1, 2, 1, 2), 48), (3, (1, 2, 4), 48), (3, (1, 2, 4), 10)])
@pytest.mark.parametrize("n", [77, 7 * 148 * 128 + 77])
def test_projected_features_of_every_layout(n, ndims, res_mode, channels, mode):
    """Gather and projection of modes 0 and 1 against fp64, one to nine pairs of 16, 32 and 48 padded channels, a partial
    tile alone and seven to eight tiles per CTA.  Bound per feature, against the sum of its terms' magnitudes: a product
    has ten roundings (three tap weights, seven of the interpolation), a projection at most six times K / 16 accumulation steps
    that need not round to nearest (2^-23).  Mode 1 with up to 152 products carries weights as one fp16 (2^-11) and
    products as two (2^-25 where the second is subnormal); with more it is fp32, as mode 0."""
    from landmark_b200.model_parallel import app_features_points

    model, sd = _pairs_model(ndims, res_mode, channels, mode)
    g = torch.Generator().manual_seed(n)
    xyz = (torch.randint(-256, 257, (n, 3), generator=g) / 256.0).cuda()
    got = app_features_points(model, xyz).double()
    ref, _ = _features_fp64(sd, ndims, len(res_mode), xyz)
    mag, w = _features_fp64(sd, ndims, len(res_mode), xyz, magnitudes=True)
    k = ndims * len(res_mode) * (-(-channels // 16) * 16)
    bound = (10 * 2.0 ** -24 + 6 * k / 16 * 2.0 ** -23) * mag + 1e-30
    if mode == 1 and k <= 152:
        bound = bound + 2.0 ** -11 * mag + 2.0 ** -25 * w.sum(1)
    worst = ((got - ref).abs() / bound).max().item()
    assert worst <= 1.0, f"error is {worst:.2f} of the bound"


@pytest.mark.parametrize("mask", [True, False])
@pytest.mark.parametrize("tables", ["negative near", "falling", "shuffled", "odd values"])
def test_hull_sampler_words_for_any_tables(tables, mask):
    """The sampler takes the tables as they are: a negative near distance (both terms rise), falling and shuffled tables,
    and tables with values that no run can be decided from.  Words equal bit for bit to testing every sample."""
    from landmark_b200._lib import check, lib
    from landmark_b200.gridnerf import B200GridNeRF

    samples, n = 133, 3001
    spec = scenes.tiny_spec().lit()
    field, ckpt = oracle_field(spec)
    if not mask:
        ckpt = {k: v for k, v in ckpt.items() if not k.startswith("alphaMask")}
    args = scenes.model_args(spec, "cuda:0")
    args.sampling_opt, args.n_importance = 1, samples
    near = -0.7 if tables == "negative near" else 0.1
    kw = dict(ckpt["kwargs"])
    kw.update({"device": "cuda:0", "args": args, "is_train": False, "near_far": (near, 6.0)})
    model = B200GridNeRF(**kw)
    model.load(ckpt)
    g = torch.Generator().manual_seed(samples)
    u = torch.linspace(0.0, 1.0, steps=samples)
    near_term = near * (1.0 - u)
    if tables == "falling":
        near_term, u = near_term.flip(0).contiguous(), u.flip(0).contiguous()
    elif tables == "shuffled":
        near_term, u = near_term[torch.randperm(samples, generator=g)], u[torch.randperm(samples, generator=g)]
    elif tables == "odd values":
        near_term[5], near_term[40], u[70], u[132] = float("nan"), float("inf"), float("nan"), -float("inf")
    if tables != "negative near":  # (that one goes through the model's own tables)
        assert model._samples(samples) == samples
        a_dev, u_dev = near_term.cuda(), u.cuda()
        check(lib.gnr_upload_hull_tables(model._handle, samples, a_dev.data_ptr(), u_dev.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
    o = torch.rand((n, 3), generator=g) * 3.0 - 1.5
    d = torch.randn((n, 3), generator=g)
    got = model.run_stages(torch.cat([o, d], 1).cuda(), samples, True, upto="sample")
    a = field.aabb.numpy()
    o, d, near_term, u = o.numpy(), d.numpy(), near_term.numpy(), u.numpy()
    with np.errstate(all="ignore"):
        far = np.where(d[:, 2] >= 0, np.float32(6.0), -((o[:, 2] - a[0, 2]) / d[:, 2]))
        z = near_term[None] + far[:, None] * u[None]
        pts = o[:, None] + d[:, None] * z[:, :, None]
        valid = snp.in_box(pts, a)
        if mask:
            m = field.alpha_aabb.numpy()
            inv = (np.float32(1.0) / (m[1] - m[0])) * np.float32(2)
            q = (pts[valid] - m[0]) * inv - np.float32(1)
            finite = np.isfinite(q).all(1)
            alpha = np.zeros(len(q), np.float32)
            alpha[finite] = snp.trilinear_zero_pad(field.alpha_volume[0, 0].numpy(), q[finite])
            at = np.nonzero(valid)
            valid[at[0][alpha <= 0], at[1][alpha <= 0]] = False
    assert pts.dtype == np.float32
    assert np.array_equal(valid_bits_from_words(got["mask_words"], samples), valid)


def test_forward_from_two_threads_returns_each_calls_status():
    """Two host threads call gnr_render_forward on one model, each with its own workspace and stream: every call returns its
    own chunk's counts and flags (one thread's list overflows, the other's does not)."""
    import threading

    from landmark_b200._lib import ST_WORDS, check, lib

    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    rays = tiny_rays(spec).cuda()
    jobs = [(rays[4800:5100].contiguous(), 64), (rays[3000:7000].contiguous(), 1)]  # rays, list entries per ray
    failures = []

    def calls(chunk, per_ray, n_calls):
        n, s = chunk.shape[0], spec.n_samples
        need = C.c_size_t(0)
        check(lib.gnr_render_workspace_bytes(model._handle, n, s, n * s, n * per_ray, C.byref(need)))
        ws = torch.empty(need.value + 256, dtype=torch.uint8, device="cuda:0")
        at = ws.data_ptr() + (-ws.data_ptr()) % 256
        rgb = torch.empty((n, 3), device="cuda:0")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        seen = []
        for _ in range(n_calls):
            st = (C.c_int32 * ST_WORDS)()
            check(lib.gnr_render_forward(model._handle, chunk.data_ptr(), n, s, 1, at, need.value, n * s, n * per_ray, rgb.data_ptr(),
                                         None, st, stream.cuda_stream))
            seen.append(tuple(st))
        return seen

    want = [calls(*job, 1)[0] for job in jobs]
    assert want[0][1] == 0 and want[1][1] == 1 and want[0][3] != want[1][3]

    def worker(i):
        try:
            failures.extend(s for s in calls(*jobs[i], 400) if s != want[i])
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=worker, args=(i % 2,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]


def test_chunk_loops_of_two_models_and_threads():
    """Chunk loops over lanes from several host threads, two models, two streams each: the lanes of a model are dealt to one
    call at a time, and no model waits for another's.  Pixels as from one thread."""
    import threading

    spec = scenes.tiny_spec().lit()
    models = [cuda_model(spec), cuda_model(spec, mlp_mode=2, app_plane_fp16=True)]
    rays = tiny_rays(spec).cuda()
    want = [m.render_rays(rays, spec.n_samples, chunk=1500, overlap=2)[0].clone() for m in models]
    torch.cuda.synchronize()
    failures = []

    def worker(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    rgb, _ = models[i % 2].render_rays(rays, spec.n_samples, chunk=1500, overlap=2)
                    if not torch.equal(rgb, want[i % 2]):
                        failures.append(i)
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]


@pytest.mark.parametrize("chunk,overlap,lanes", [(500, 12, 8), (5000, 6, 2), (4000, 3, 3), (20000, 4, 1), (500, 1, 1), (500, True, 2)])
def test_any_number_of_lanes_is_accepted(chunk, overlap, lanes):
    """More side streams than the library has lanes, or than there are chunks: same pixels, a workspace per lane in use."""
    from landmark_b200._lib import MAX_LANES

    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    rays = tiny_rays(spec).cuda()
    want, _ = model.render_rays(rays, spec.n_samples, chunk=10000)
    model.release_workspaces()
    got, _ = model.render_rays(rays, spec.n_samples, chunk=chunk, overlap=overlap)
    assert torch.equal(got, want) and len(model._ws) == lanes <= MAX_LANES


def test_status_of_an_empty_chunk_loop_is_its_own():
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    rays = tiny_rays(spec).cuda()
    model.app_capacity_per_ray = 1
    model.render_rays(rays, spec.n_samples)
    assert model.render_rays(rays[:0], spec.n_samples)[0].shape == (0, 3)
    assert not model.check_pending_status().any()


def _runners(model, spec, sizes, **kw):
    """Runners of one renderer, an image size each."""
    from landmark_b200.engine import FrameRenderer, NerfDDPRunner

    renderer = FrameRenderer(model, spec.n_samples, **kw)
    return [NerfDDPRunner(renderer, h, w, focal=spec.focal) for h, w in sizes]


def test_frames_of_one_renderer_on_two_streams():
    """Two runners share a renderer and enqueue frames of their own poses on a stream each, nothing waited for in between:
    every image is that of its pose."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec, mlp_mode=2, app_plane_fp16=True)
    runners = _runners(model, spec, [(100, 100), (100, 100)], chunk=3000)
    poses = [scenes.look_at((1.2, 1.2, 1.0), (0.0, 0.0, 0.0)), scenes.look_at((-1.0, 1.4, 0.8), (0.0, 0.0, 0.0))]
    want = [r.run_batch(p).copy() for r, p in zip(runners, poses)]
    assert not np.array_equal(*want)
    streams = [torch.cuda.Stream() for _ in runners]
    images = [[torch.zeros((100, 100, 4), dtype=torch.uint8).pin_memory() for _ in range(30)] for _ in runners]
    for k in range(30):
        for r, p, s, im in zip(runners, poses, streams, images):
            with torch.cuda.stream(s):
                r.enqueue(p, im[k])
    torch.cuda.synchronize()
    for w, im in zip(want, images):
        assert all(np.array_equal(w, i.numpy()) for i in im)
    runners[0].renderer.finish()


def test_frames_of_changing_size_wait_for_nothing(monkeypatch):
    """A renderer that alternates between image sizes and chunk counts: no device-wide wait, and no new pinned memory once
    every slot has been used."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    runners = _runners(model, spec, [(100, 100), (90, 70), (30, 30)])
    pose = scenes.make_pose(spec)
    want = [r.run_batch(pose).copy() for _ in range(8) for r in runners][-3:]

    def fail(*a, **k):
        raise AssertionError("waits or pins memory")

    monkeypatch.setattr(torch.cuda, "synchronize", fail)
    monkeypatch.setattr(torch.Tensor, "pin_memory", fail)
    for _ in range(4):
        for r, w in zip(runners, want):
            assert np.array_equal(r.run_batch(pose), w)


def test_whole_frame_leaves_the_colours_in_the_runner():
    """``rgb`` (tile order) and ``image`` (row order) of a runner hold the frame in fp32, as the stages leave them."""
    from landmark_b200.engine import FrameRenderer, NerfDDPRunner

    class Stages(FrameRenderer):
        def to_rgba8(self, image, out):
            super().to_rgba8(image, out)

    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    for pose in (scenes.make_pose(spec), scenes.look_at((1.2, 1.2, 1.0), (0.0, 0.0, 0.0))):
        for h, w in ((100, 100), (37, 61)):
            whole, staged = (NerfDDPRunner(r(model, spec.n_samples, chunk=3000), h, w, focal=spec.focal) for r in (FrameRenderer, Stages))
            assert np.array_equal(whole.run_batch(pose), staged.run_batch(pose))
            assert torch.equal(whole.rgb, staged.rgb) and torch.equal(whole.image, staged.image) and whole.image.std() > 0


def test_frame_call_checks_its_arguments():
    """Pixel lists of any integer type are converted, as generate_rays does; buffers of another type, size or place, which
    the library would write as raw memory, are refused."""
    from landmark_b200.engine import FrameRenderer
    from landmark_b200.rays import device_tables

    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    runner = _runners(model, spec, [(60, 50)])[0]
    pose = scenes.make_pose(spec)
    want = runner.run_batch(pose).copy()
    ids = runner.shard.pixel_ids
    renderer = FrameRenderer(model, spec.n_samples)
    for other in (ids.to(torch.int64), ids.cpu(), torch.stack([ids, ids], 1)[:, 0]):
        image = torch.zeros((60, 50, 4), dtype=torch.uint8).pin_memory()
        renderer.render_frame(pose, 60, 50, spec.focal, other, runner.rgba, image).synchronize()
        assert np.array_equal(want, image.numpy())
    dev = {"device": "cuda:0"}
    good = {"rays": torch.empty((3000, 6), **dev), "rgba": torch.empty((3000, 4), dtype=torch.uint8, **dev),
            "host_image": torch.empty((60, 50, 4), dtype=torch.uint8).pin_memory(), "status": torch.empty((1, 8), dtype=torch.int32).pin_memory(),
            "rgb": torch.empty((3000, 3), **dev), "image": torch.empty((3000, 3), **dev), "pixel_ids": ids, "pose": pose}

    def call(**changed):
        a = dict(good, **changed)
        model.render_frame(a["pose"], device_tables(60, 50, spec.focal, "cuda:0"), 60, 50, a["pixel_ids"], spec.n_samples, True, 131072, 2,
                           a["rays"], a["rgba"], a["host_image"], a["status"], a["rgb"], a["image"])

    call()
    torch.cuda.synchronize()
    assert np.array_equal(want, good["host_image"].numpy())
    for changed in ({"rays": good["rays"].half()}, {"rays": good["rays"][:-1]}, {"rays": good["rays"].cpu()}, {"rgba": good["rgb"]},
                    {"rgba": torch.empty((60, 100, 4), dtype=torch.uint8, **dev)[:, ::2]}, {"host_image": good["host_image"].clone()},
                    {"host_image": good["rgba"]}, {"status": good["status"].clone()}, {"status": good["status"][:0]},
                    {"rgb": good["rgb"].double()}, {"image": good["image"][1:]}, {"pixel_ids": ids[:-1]}, {"pose": pose[:2]}):
        with pytest.raises(ValueError):
            call(**changed)


def test_stages_replaced_on_objects_are_run():
    """A renderer whose stages, or a model whose chunk loop, are replaced in a subclass or on the object: the frame goes
    through them."""
    from landmark_b200.gridnerf import B200GridNeRF

    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    pose = scenes.make_pose(spec)
    runner = _runners(model, spec, [(30, 30)])[0]
    want = runner.run_batch(pose).copy()
    ran = []

    def noting(name, stage):
        def f(*a, **k):
            ran.append(name)
            return stage(*a, **k)
        return f

    for obj, name in ((runner.renderer, "render_pixels"), (runner.renderer, "to_rgba8"), (model, "render_rays")):
        setattr(obj, name, noting(name, getattr(obj, name)))
        assert np.array_equal(runner.run_batch(pose), want) and ran[-1] == name
        delattr(obj, name)

    class Own(B200GridNeRF):
        def render_rays(self, *a, **k):
            ran.append("subclass")
            return super().render_rays(*a, **k)

    model.__class__ = Own
    assert np.array_equal(runner.run_batch(pose), want) and ran[-1] == "subclass"


def test_frame_with_a_chunk_size_below_one():
    """Chunk sizes below one ray mean one ray, as in the chunk loop."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    pose = scenes.make_pose(spec)
    want = _runners(model, spec, [(7, 9)])[0].run_batch(pose)
    for chunk in (0, -3):
        assert np.array_equal(_runners(model, spec, [(7, 9)], chunk=chunk)[0].run_batch(pose), want)


def test_a_frame_can_be_captured():
    """enqueue under a CUDA graph capture goes stage by stage, which a graph can replay."""
    spec = scenes.tiny_spec().lit()
    model = cuda_model(spec)
    pose = scenes.make_pose(spec)
    runner = _runners(model, spec, [(50, 50)])[0]
    want = runner.run_batch(pose).copy()
    image = torch.zeros((50, 50, 4), dtype=torch.uint8).pin_memory()
    model.render_rays(runner.rgb.new_zeros((2500, 6)), spec.n_samples)  # (workspace)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        runner.enqueue(pose, image)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(image.numpy(), want)


def _inferer(spec, chunk, **options):
    from types import SimpleNamespace

    from landmark_b200.inferer import B200NerfDDPInfererImpl

    args = scenes.model_args(spec, "cuda:0")
    args.render_batch_size = chunk
    impl = B200NerfDDPInfererImpl(SimpleNamespace(args_nerf=args, checkpoint=scenes.make_checkpoint(spec), model_path=None), **options)
    impl.load_model(spec.height, spec.width)
    return impl


def test_inferer_runs_what_is_hooked_to_the_forward():
    """Forward hooks of the model, global ones, and a forward replaced on the object or in a subclass run once per chunk of
    render_batch_size rays, as in the plain chunk loop."""
    from landmark_b200.gridnerf import B200GridNeRF

    spec = scenes.tiny_spec().lit()
    impl = _inferer(spec, 2048)
    model = impl.model
    rays = tiny_rays(spec).cuda()
    want = impl.renderer_fn(rays, N_samples=spec.n_samples)
    ran = []

    def count(*a, **k):
        ran.append(1)

    for register in (model.register_forward_hook, model.register_forward_pre_hook,
                     torch.nn.modules.module.register_module_forward_hook, torch.nn.modules.module.register_module_forward_pre_hook):
        ran.clear()
        handle = register(count)
        assert torch.equal(impl.renderer_fn(rays, N_samples=spec.n_samples), want)
        handle.remove()
        assert len(ran) == 5
    ran.clear()
    forward = model.forward
    model.forward = lambda *a, **k: (count(), forward(*a, **k))[1]
    assert torch.equal(impl.renderer_fn(rays, N_samples=spec.n_samples), want) and len(ran) == 5
    del model.forward

    class Own(B200GridNeRF):
        def forward(self, *a, **k):
            count()
            return super().forward(*a, **k)

    ran.clear()
    model.__class__ = Own
    assert torch.equal(impl.renderer_fn(rays, N_samples=spec.n_samples), want) and len(ran) == 5


def test_inferer_without_status_checks():
    """With ``check_status_every_call`` off renderer_fn neither waits for the status nor raises, as its chunks' forwards; the
    status is there to be asked for."""
    spec = scenes.tiny_spec().lit()
    impl = _inferer(spec, 2048)
    rays = tiny_rays(spec).cuda()
    impl.model.app_capacity_per_ray = 1
    with pytest.raises(RuntimeError, match="appearance-sample list overflow"):
        impl.renderer_fn(rays, N_samples=spec.n_samples)
    impl.model.check_status_every_call = False
    assert impl.renderer_fn(rays, N_samples=spec.n_samples).shape == (10000, 3)
    with pytest.raises(RuntimeError, match="appearance-sample list overflow"):
        impl.model.check_pending_status()


def test_inferer_stays_within_memory(monkeypatch):
    """render_batch_size is what a caller sized its memory for: larger device chunks are taken only where their workspaces
    are a small share of the free memory, and given up when an allocation fails.  Same pixels."""
    spec = scenes.tiny_spec().lit()
    rays = tiny_rays(spec).cuda()
    impl = _inferer(spec, 1000)
    model = impl.model
    one = model.workspace_bytes(1000, spec.n_samples)
    assert impl._device_chunk(10000, spec.n_samples) == (65536, 1) and impl._device_chunk(200000, spec.n_samples) == (65536, 2)
    want = impl.renderer_fn(rays, N_samples=spec.n_samples)
    impl.RENDER_UNASKED = 0
    for share, lanes in ((20.0, 1), (3.0, 2), (0.5, 1)):  # free memory in workspaces of 1000 rays
        model.release_workspaces()
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (int(8 * share * one), 1 << 40))
        assert torch.equal(impl.renderer_fn(rays, N_samples=spec.n_samples), want)
        held = sum(w.numel() for w in model._ws.values())
        assert len(model._ws) == lanes and held <= max(share, 1.0) * one + 1024, (share, held / one)
    monkeypatch.undo()
    model.release_workspaces()
    made = model.workspace

    def no_room(n, *a, **k):
        if n > 1000:
            raise torch.cuda.OutOfMemoryError("no room")
        return made(n, *a, **k)

    monkeypatch.setattr(model, "workspace", no_room)
    for _ in range(2):
        assert torch.equal(impl.renderer_fn(rays, N_samples=spec.n_samples), want)
        assert len(model._ws) == 1 and model._ws[0].numel() <= one + 512
    monkeypatch.setattr(model, "workspace", lambda *a, **k: no_room(1001))
    with pytest.raises(torch.cuda.OutOfMemoryError):
        impl.renderer_fn(rays, N_samples=spec.n_samples)


def test_sampler_words_in_a_mask_longer_than_its_floats():
    """A mask of 2 x 2 x (2^23 + 2^21) cells, where the index of a far sample has no fraction left: words as the test of
    every sample gives them."""
    from landmark_b200.gridnerf import AlphaGridMask, B200GridNeRF

    spec = scenes.tiny_spec(grid=16).lit()
    ckpt = scenes.make_checkpoint(spec)
    kw = dict(ckpt["kwargs"])
    kw.update({"device": "cuda:0", "args": scenes.model_args(spec, "cuda:0"), "is_train": False})
    model = B200GridNeRF(**kw)
    width = (1 << 23) + (1 << 21)
    g = torch.Generator().manual_seed(5)
    volume = (torch.rand((2, 2, width), generator=g) < 0.1)
    model.alphaMask = AlphaGridMask(torch.device("cuda:0"), ckpt["alphaMask.aabb"].cuda(), volume.float().cuda())
    model.load({k: v for k, v in ckpt.items() if not k.startswith("alphaMask")})
    n, samples = 2000, 64
    o = torch.rand((n, 3), generator=g) * 2.0 - 1.0
    d = torch.randn((n, 3), generator=g) * torch.tensor([1.0, 0.1, 0.1])
    got = model.run_stages(torch.cat([o, d], 1).cuda(), samples, True, upto="sample")
    field, _ = oracle_field(spec)
    valid, _ = snp.valid_mask(torch.cat([o, d], 1).numpy(), field.aabb.numpy(), field.near, field.far, field.step_size.item(), samples,
                              volume.float().numpy(), field.alpha_aabb.numpy(), 0.0)
    assert 0.05 < valid.mean() < 0.95
    assert np.array_equal(valid_bits_from_words(got["mask_words"], samples), valid)

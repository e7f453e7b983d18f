"""GPU tests of single kernels at the sizes where their work split has its edges: partial tiles and words, the
smallest and largest chunk a rule picks a form for.  References: the CPU oracle, or the same pixels computed another way."""
import numpy as np
import pytest
import torch

from landmark_b200 import scenes
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

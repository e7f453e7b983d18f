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

"""Seed lists of masked Voronoi labelling that hold a large part of the image, as the
eroded masks of eroded_otsu_labeling do."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cle():
    import pyclesperanto_prototype_b200 as m
    from pyclesperanto_prototype_b200 import _build
    _build.build()
    return m


# voxel counts on both sides of the one-launch form's limits (2^15 here, 2^17 for
# maxima), seeds from none to every voxel of the mask
@pytest.mark.parametrize("shape", [(31, 33), (181, 181), (182, 181), (16, 32, 64), (17, 32, 64), (362, 362), (32, 64, 64),
                                   (33, 64, 64)])
@pytest.mark.parametrize("fill", [0.0, 0.02, 0.4, 1.0])
def test_masks_as_their_own_seeds(cle, oracle, shape, fill):
    r = np.random.default_rng(17)
    mask = (r.uniform(size=shape) < fill).astype(np.uint8)
    for seeds in (mask, mask * (r.uniform(size=shape) < 0.5)):
        seeds = seeds.astype(np.uint8)
        got = cle.pull(cle.masked_voronoi_labeling_binary(cle.push_native(seeds), cle.push_native(mask)))
        assert np.array_equal(got, oracle.masked_voronoi_labeling(seeds, mask))


# the voxels of a plateau from 2^24 on are all maxima (v - 1 == v): the list of
# voronoi_otsu_labeling can be dense as well
@pytest.mark.parametrize("shape", [(120, 200), (20, 60, 70)])
def test_plateaus_of_large_values(cle, oracle, shape):
    a = np.zeros(shape, np.float32)
    a[tuple(slice(s // 4, -s // 4) for s in shape)] = 2.0 ** 27
    got = cle.pull(cle.voronoi_otsu_labeling(a, spot_sigma=0, outline_sigma=0))
    assert np.array_equal(got, oracle.voronoi_otsu_labeling(a, 0, 0))


# a mask's voxels as seeds cost about as much just below the line (one launch) as
# above it; with the unions of the list in one CTA it was 18 times as much
def test_dense_seeds_are_not_left_to_one_cta(cle):
    times = []
    for shape in ((32, 64, 64), (34, 64, 64)):
        mask = cle.push_native((np.random.default_rng(3).uniform(size=shape) < 0.9).astype(np.uint8))
        out = cle.create_labels_like(mask)
        best = []
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            cle.masked_voronoi_labeling_binary(mask, mask, out)
            e1.record()
            torch.cuda.synchronize()
            best.append(e0.elapsed_time(e1))
        times.append(min(best))
    assert times[0] < 3 * times[1]

"""Growth over the whole image whose paths pass the step range of the key growth,
which then hands the labels back to the step-by-step growth."""
import time

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


def _seeds(shape, density, seed):
    r = np.random.default_rng(seed)
    lab = np.where(r.uniform(size=shape) < density, r.integers(1, 100000, size=shape), 0).astype(np.uint32)
    lab.reshape(-1)[0] = 1
    return lab


# whether paths get too long shows in the middle of a round, to one block before
# another: every block has to leave the rounds at the same one, or the rest wait at a
# barrier for blocks that have gone (4 s for this call, when the word that says so was
# read while it could still be set)
@pytest.mark.parametrize("shape,density", [((1024, 1024), 3e-4), ((1024, 1024), 2e-4), ((700, 900), 2.5e-4), ((2048, 2048), 3e-4)])
@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_paths_beyond_the_step_range(cle, oracle, shape, density, seed):
    lab = _seeds(shape, density, seed)
    dev = cle.B200Array(torch.from_numpy(lab.astype(np.int32)).cuda().view(torch.uint32))
    out = cle.extend_labeling_via_voronoi(dev)
    if shape == (700, 900):
        assert np.array_equal(cle.pull(out).astype(np.uint32), oracle.extend_labeling_via_voronoi(lab))
    first = cle.pull(out)
    for _ in range(6):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        cle.extend_labeling_via_voronoi(dev, out)
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 1.0
        assert np.array_equal(cle.pull(out), first)


@pytest.mark.parametrize("shape,seeds", [((300, 260), 1), ((300, 260), 9), ((20, 150, 170), 2), ((150, 150), 3)])
def test_few_seeds(cle, oracle, shape, seeds):
    lab = np.zeros(shape, np.uint32)
    r = np.random.default_rng(5)
    lab.reshape(-1)[r.choice(lab.size, seeds, replace=False)] = np.arange(1, seeds + 1)
    dev = cle.B200Array(torch.from_numpy(lab.astype(np.int32)).cuda().view(torch.uint32))
    assert np.array_equal(cle.pull(cle.extend_labeling_via_voronoi(dev)).astype(np.uint32), oracle.extend_labeling_via_voronoi(lab))


# labels in nearly every 8 x 4 (x 4) brick: the step-by-step growth takes over; one brick in 512
# empty, two, none, images with partial bricks
@pytest.mark.parametrize("shape", [(64, 128), (64, 256), (61, 250), (16, 64, 64), (15, 62, 61), (1, 8, 70), (40, 3, 5)])
@pytest.mark.parametrize("empty", [0, 1, 2, 3])
def test_labels_in_nearly_every_brick(cle, oracle, shape, empty):
    r = np.random.default_rng(6)
    lab = np.where(r.uniform(size=shape) < 0.5, r.integers(1, 1000, size=shape), 0).astype(np.uint32)
    for k in range(empty):
        x = 8 * (2 * k) % (8 * (-(-shape[-1] // 8)))
        lab[..., :4, x:x + 8][..., :, :] = 0 if len(shape) == 2 else lab[..., :4, x:x + 8]
        if len(shape) == 3:
            lab[:4, :4, x:x + 8] = 0
    if lab.max() == 0:
        lab.reshape(-1)[-1] = 5
    for src in (cle.B200Array(torch.from_numpy(lab.astype(np.int32)).cuda().view(torch.uint32)), lab.astype(np.float32)):
        assert np.array_equal(cle.pull(cle.extend_labeling_via_voronoi(src)).astype(np.uint32), oracle.extend_labeling_via_voronoi(lab))

"""Connected components on both sides of the lines between the forms of the
labelling (row runs for small and thin images, tiles otherwise)."""
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


def _mask(shape, kind, seed=21):
    r = np.random.default_rng(seed)
    if kind == "snake":          # one object whose runs link up in a long chain
        m = np.zeros(shape, bool)
        m[..., ::2, :] = True
        m[..., 1::4, -1:] = True
        m[..., 3::4, :1] = True
        return m.astype(np.uint8)
    return (r.uniform(size=shape) < kind).astype(np.uint8)


# 2^20 pixels, 3 x 2^18 voxels (2^20 with face connectivity), and the number of rows against the rows of the tiles
SHAPES = [(1, 1), (3, 70), (1024, 1024), (1025, 1024), (8, 131500), (9, 131500), (1, 1200000), (48, 128, 128), (49, 128, 128),
          (64, 128, 128), (65, 128, 128),
          (4, 2, 70000), (9, 2, 40000), (17000, 1, 32), (17000, 2, 16), (64, 90, 91)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", [0.1, 0.35, 0.6, 1.0, "snake"])
def test_labels_of_both_forms(cle, oracle, shape, kind):
    m = _mask(shape, kind)
    got = cle.pull(cle.connected_components_labeling_box(cle.push_native(m)))
    assert np.array_equal(got, oracle.connected_components_labeling_box(m))
    got = cle.pull(cle.connected_components_labeling_diamond(cle.push_native(m)))
    assert np.array_equal(got, oracle.connected_components_labeling_diamond(m))


@pytest.mark.parametrize("shape", [(200, 333), (1030, 1024), (20, 33, 65), (40, 130, 128)])
def test_labels_in_place_and_of_other_types(cle, oracle, shape):
    m = _mask(shape, 0.4)
    want = oracle.connected_components_labeling_box(m)
    for dtype in (torch.uint32, torch.float32):
        a = cle.B200Array(torch.from_numpy(m.astype(np.int32)).cuda().to(dtype))
        cle.connected_components_labeling_box(a, a)
        assert np.array_equal(cle.pull(a).astype(np.uint32), want)
    f = (m * np.float32(-2.5)).astype(np.float32)      # anything but zero is foreground
    assert np.array_equal(cle.pull(cle.connected_components_labeling_box(f)), want)


@pytest.mark.parametrize("shape", [(300, 400), (1030, 1030), (20, 64, 64), (40, 130, 130)])
def test_gauss_otsu_of_both_forms(cle, oracle, shape):
    a = np.random.default_rng(4).uniform(0, 1000, size=shape).astype(np.float32)
    assert np.array_equal(cle.pull(cle.gauss_otsu_labeling(a, outline_sigma=1.0)), oracle.gauss_otsu_labeling(a, 1.0))


def _time(cle, shape, fill):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    m = cle.B200Array((torch.rand(shape, generator=g, device="cuda") < fill).to(torch.uint8))
    out = cle.create_labels_like(m)
    best = []
    for _ in range(8):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(10):
            cle.connected_components_labeling_box(m, out)
        e1.record()
        torch.cuda.synchronize()
        best.append(e0.elapsed_time(e1))
    return min(best)


# tiles for every image made one row of 4M pixels 6 times as slow as 2048 x 2048 and a
# volume of 1/8 of the voxels nearly as slow as the whole
def test_small_and_thin_images_are_not_left_to_tiles(cle):
    assert _time(cle, (1, 1 << 22), 0.1) < 2 * _time(cle, (2048, 2048), 0.1)
    assert _time(cle, (32, 64, 64), 0.5) < 0.6 * _time(cle, (64, 128, 128), 0.5)

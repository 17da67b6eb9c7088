"""Images longer along one axis than a CUDA grid's second and third axes reach
(65535), and destinations that start in the middle of an allocation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cle():
    import pyclesperanto_prototype_b200 as m
    from pyclesperanto_prototype_b200 import _build
    _build.build()
    return m


def _image(shape, dtype, seed=5):
    return np.random.default_rng(seed).integers(0, 60000, size=shape).astype(dtype)


# radius 12 takes the three-pass form, 8 the fused one; the y pass of a volume runs
# over all its planes at once, a long image has many tiles along y
@pytest.mark.parametrize("shape,sigma", [((65537, 2, 3), (3, 3, 3)), ((65537, 2, 4), (3, 3, 3)), ((65537, 2, 3), (2, 2, 2)),
                                         ((70000, 3, 1), (0, 1, 0.5)), ((65536 * 128 + 1, 1), (0, 1.5, 0))])
@pytest.mark.parametrize("dtype", [np.uint16, np.float32])
def test_gaussian_blur_of_long_axes(cle, oracle, shape, sigma, dtype):
    a = _image(shape, dtype)
    got = cle.pull(cle.gaussian_blur(a, None, *sigma))
    assert np.array_equal(got, oracle.gaussian_blur(a.astype(np.float32), *sigma))


@pytest.mark.parametrize("sigma", [2.0, 3.0])
def test_labelings_of_many_planes(cle, oracle, sigma):
    a = _image((65537, 2, 3), np.uint16)
    f = a.astype(np.float32)
    assert np.array_equal(cle.pull(cle.gauss_otsu_labeling(a, outline_sigma=sigma)), oracle.gauss_otsu_labeling(f, sigma))
    for spot, outline in ((sigma, sigma), (1.0, sigma), (sigma, 1.0)):
        got = cle.pull(cle.voronoi_otsu_labeling(a, spot_sigma=spot, outline_sigma=outline))
        assert np.array_equal(got, oracle.voronoi_otsu_labeling(f, spot, outline))


# a destination (and a source) that starts one element into its allocation, with
# rows whose length alone would allow wide loads and stores
@pytest.mark.parametrize("shape", [(40, 64), (7, 36, 64), (3, 5, 6)])
@pytest.mark.parametrize("sigma", [(0.5, 0.5, 0.5), (2, 2, 2), (3.5, 3.5, 3.5), (1, 2, 0.5)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
def test_gaussian_blur_of_views_off_alignment(cle, oracle, shape, sigma, dtype):
    import torch
    n = int(np.prod(shape))
    a = np.random.default_rng(6).integers(0, 255, size=shape).astype(dtype)
    src = torch.zeros(n + 1, dtype=getattr(torch, np.dtype(dtype).name), device="cuda")
    src[1:].copy_(torch.from_numpy(a.reshape(-1)))
    buf = torch.full((n + 3,), -1.0, device="cuda")
    dst = cle.B200Array(buf[1:1 + n].view(shape))
    cle.gaussian_blur(cle.B200Array(src[1:].view(shape)), dst, *sigma)
    assert np.array_equal(cle.pull(dst), oracle.gaussian_blur(a.astype(np.float32), *sigma))
    assert buf[0].item() == -1.0 and buf[-2:].eq(-1.0).all()


# widths and heights on both sides of the tile counts from which volumes are staged
# by TMA copies (8 x 8 tiles of 32 x 32 for 8/16-bit sources, 16 x 16 for float32)
@pytest.mark.parametrize("dtype,width,height", [(np.uint8, 224, 256), (np.uint8, 240, 225), (np.uint16, 232, 224),
                                                (np.uint16, 256, 250), (np.float32, 480, 481), (np.float32, 484, 481),
                                                (np.float32, 512, 500)])
@pytest.mark.parametrize("depth,sigma", [(1, 0.5), (3, 2.0), (9, 1.0), (21, 2.0)])
def test_gaussian_blur_either_side_of_tma_staging(cle, oracle, dtype, width, height, depth, sigma):
    a = np.random.default_rng(8).integers(0, 255, size=(depth, height, width)).astype(dtype)
    got = cle.pull(cle.gaussian_blur(a, None, sigma, sigma, sigma))
    assert np.array_equal(got, oracle.gaussian_blur(a.astype(np.float32), sigma, sigma, sigma))


# a source that could be staged by TMA copies (16-byte aligned) is not slower than
# the same one element further, which cannot (narrow and small volumes: 1.4 to 1.8
# times the time while they were staged by TMA)
@pytest.mark.parametrize("shape", [(16, 16, 16), (512, 8, 8), (512, 1024, 16), (128, 512, 512)])
@pytest.mark.parametrize("dtype", ["uint16", "float32"])
def test_aligned_sources_are_not_slower(cle, shape, dtype):
    import torch
    from pyclesperanto_prototype_b200 import _lib
    lib, n = _lib.load(), int(np.prod(shape))
    buf = torch.randint(0, 1000, (n + 1,), device="cuda", dtype=torch.int32).to(getattr(torch, dtype))
    out = torch.empty(shape, device="cuda")
    best = []
    for src in (buf[:n].view(shape), buf[1:].view(shape)):
        s, d = _lib.tensor_desc(src), _lib.tensor_desc(out)
        ws = torch.empty(lib.cle_gaussian_blur_workspace_bytes(_lib.ref(s)), dtype=torch.uint8, device="cuda")
        args = (_lib.ref(s), _lib.ref(d), 2.0, 2.0, 2.0, ws.data_ptr(), ws.numel(), _lib.stream_ptr())
        times = []
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(40):
                _lib.check(lib.cle_gaussian_blur(*args))
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        best.append(min(times))
    assert best[0] <= 1.25 * best[1]


# the status word of a volume's blur, whichever form it takes and whatever the
# workspace held; an axis without a blur ends the three-pass form with a copy
@pytest.mark.parametrize("sigma", [(2, 2, 2), (3, 3, 3), (1, 2, 0.5), (4, 0, 0), (0, 0, 4), (0, 0, 0)])
@pytest.mark.parametrize("shape", [(5, 40, 48), (9, 260, 272)])
def test_status_word_of_a_blur(cle, oracle, shape, sigma):
    import torch
    from pyclesperanto_prototype_b200 import _lib
    lib = _lib.load()
    a = _image(shape, np.uint16)
    src, dst = torch.from_numpy(a).cuda(), torch.empty(shape, device="cuda")
    s, d = _lib.tensor_desc(src), _lib.tensor_desc(dst)
    ws = torch.full((lib.cle_gaussian_blur_workspace_bytes(_lib.ref(s)),), 255, dtype=torch.uint8, device="cuda")
    stream = _lib.stream_ptr()
    _lib.check(lib.cle_gaussian_blur(_lib.ref(s), _lib.ref(d), *[float(v) for v in sigma], ws.data_ptr(), ws.numel(), stream))
    assert lib.cle_workspace_status(ws.data_ptr(), ws.numel(), stream) == 0
    assert np.array_equal(dst.cpu().numpy(), oracle.gaussian_blur(a.astype(np.float32), *sigma))


# rows split over fewer or more row pairs per CTA: few rows, long windows
@pytest.mark.parametrize("shape", [(1, 256), (2, 300), (9, 40), (700, 24), (5, 7, 33)])
@pytest.mark.parametrize("sigma", [(100, 0.5, 0), (20, 0, 3), (6, 7, 8)])
def test_gaussian_blur_of_few_rows(cle, oracle, shape, sigma):
    a = _image(shape, np.uint16)
    got = cle.pull(cle.gaussian_blur(a, None, *sigma))
    assert np.array_equal(got, oracle.gaussian_blur(a.astype(np.float32), *sigma))

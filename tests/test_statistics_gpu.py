"""Statistics of labels: totals beyond float64's integers, images of many small
labels."""
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


def _total_of(target, width):
    """uint16 intensities of one row whose sum of intensity * x is `target`: all terms
    multiples of 4 except one."""
    v = np.zeros(width, np.uint16)
    rest = target // 4
    for x in range(width - 1, 0, -1):
        k = min(16383, rest // x)
        v[x] = 4 * k
        rest -= k * x
        if rest == 0:
            break
    assert rest == 0
    v[1] += target % 4
    return v


def _on_device(cle, labels):
    return cle.B200Array(torch.from_numpy(labels.astype(np.int32)).cuda().view(torch.uint32))


# one above the middle of two float32 values above 2^53: a total that drops its last
# bit on the way (as float64 does there) rounds to the lower one
@pytest.mark.parametrize("axis", ["x", "y"])
def test_totals_beyond_2_to_53_are_exact(cle, axis):
    target = 2 ** 53 + 2 ** 29 + 1
    row = _total_of(target, 1 << 20)
    assert int(np.sum(row.astype(object) * np.arange(row.size))) == target
    image = np.ascontiguousarray(row[None, :] if axis == "x" else row[:, None])
    table = cle.statistics_of_labelled_pixels(cle.push_native(image), _on_device(cle, np.ones(image.shape)))
    assert float(table["sum_intensity_times_" + axis][0]) == 2 ** 53 + 2 ** 30

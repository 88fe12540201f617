"""Slices cut from a spectrum into images of more tiles along an axis than a
grid's y or z dimension holds."""
import numpy as np
import pytest

from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import spectrum_and_views

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small", [((1 << 22, 4), (64, 4)), ((4, 1 << 21), (4, 64))])
def test_images_of_many_tiles(large, small):
    """The same few frequencies in a larger image: its samples at the smaller
    one's places are the same sums.  Both transforms are FP32: 1e-5 of the
    largest sample is the suite's tolerance."""
    rng = np.random.default_rng(5)
    cons = constraints(rng.random((500, 3), dtype=np.float32), rng.standard_normal(500).astype(np.float32))
    cutoff = tuple(min(16, s // 2) for s in small)
    views = [((1, 0, 0), (0, 1, 0)), ((0.6, 0.0, 0.8), (0, 1, 0))]
    images = [spectrum_and_views([(cons, None, M.WENDLAND_D3_C2)], (32, 32, 32), 1.0, (1.0, 1.0), cutoff, samples,
                                 views, M.FORM_PLAIN)[1] for samples in (large, small)]
    at_small = images[0][:, ::large[0] // small[0], ::large[1] // small[1]]
    assert np.max(np.abs(at_small - images[1])) < 1e-5 * np.max(np.abs(images[1]))

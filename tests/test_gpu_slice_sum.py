"""The direct slice's own kernels (register-tiled product of separable groups;
table kernel of SPH and Wendland groups with varying radii on square slices)
and its finalize, against the FP64 oracle: cutoffs around the tiles (4 x values,
64 representatives), particle counts around a stage, a tile and a split, and
the routes to the folded form (a slice that is not square)."""
import numpy as np
import pytest

import oracle as O
from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import render_direct

pytestmark = pytest.mark.gpu

TOL = 1e-5  # the direct slice's tolerance (rel-L2), as for the other direct renders

U, V = (0.8, 0.0, -0.6), (0.0, 1.0, 0.0)


def _group(rng, n, basis, radii, scale):
    p = rng.random((n, 3), dtype=np.float32)
    w = rng.standard_normal(n).astype(np.float32)
    h = {"none": None, "uniform": np.full(n, scale, np.float32),
         "varying": rng.uniform(0.1 * scale, scale, n).astype(np.float32)}[radii]
    return constraints(p, w), h, basis


def _check(groups, cutoff, samples, step=(1.0, 1.0), partial_sums=1):
    img = render_direct(groups, step, cutoff, U, V, samples, partial_sums=partial_sums)
    ref = O.render_direct(groups, step, cutoff, U, V, samples)
    assert O.rel_l2(img, ref) < TOL


# cutoffs whose 2 c^2 is a multiple of the block length (64)
@pytest.mark.parametrize("cutoff", [8, 16, 40, 64, 72])
@pytest.mark.parametrize("radii", ["none", "uniform", "varying"])
@pytest.mark.parametrize("basis", [M.SPH, M.WENDLAND_D3_C2, M.GAUSSIAN, M.GAUSSIAN_DECAYING])
def test_square_slices(basis, radii, cutoff):
    if basis == M.GAUSSIAN and radii == "none":
        pytest.skip("exp(+pi |k|^2) exceeds the float range")
    rng = np.random.default_rng(cutoff)
    scale = (1.0 if basis == M.GAUSSIAN else 3.0) / (1.5 * cutoff)
    _check([_group(rng, 1500, basis, radii, scale)], (cutoff, cutoff), (2 * cutoff + 3, 2 * cutoff + 2))


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 255, 257, 20011])
@pytest.mark.parametrize("basis,radii", [(M.SPH, "none"), (M.WENDLAND_D3_C2, "varying"),
                                         (M.GAUSSIAN_DECAYING, "varying")])
def test_particle_counts(n, basis, radii):
    _check([_group(np.random.default_rng(n), n, basis, radii, 0.05)], (24, 24), (48, 49))


@pytest.mark.parametrize("radii", ["none", "varying"])
@pytest.mark.parametrize("basis", [M.SPH, M.GAUSSIAN_DECAYING])
def test_slices_that_are_not_square_and_several_groups(basis, radii):
    rng = np.random.default_rng(3)
    groups = [_group(rng, 700, basis, radii, 0.04), _group(rng, 0, basis, radii, 0.04),
              _group(rng, 300, M.WENDLAND_D3_C2, "varying", 0.05)]
    _check(groups, (16, 40), (37, 90), partial_sums=2)
    _check(groups, (24, 24), (48, 60), step=(0.5, 0.75))
    _check(groups, (24, 24), (50, 48), step=(0.5, 0.5))


def test_radii_past_the_table_and_zero_radii():
    """|k| h beyond the last cell (Phi^ there is below 1e-11) and zero radii."""
    rng = np.random.default_rng(4)
    c, h, b = _group(rng, 600, M.WENDLAND_D3_C2, "varying", 0.05)
    h[::7] = 5.0
    h[3::11] = 0.0
    _check([(c, h, b)], (32, 32), (64, 64))


@pytest.mark.parametrize("basis", [M.SPH, M.WENDLAND_D3_C2, M.GAUSSIAN_DECAYING])
@pytest.mark.parametrize("n", [300, 8192])  # statistics from the host, from the device
@pytest.mark.parametrize("cutoff", [(16, 16), (16, 40)])
def test_a_nan_among_equal_radii_shows(basis, n, cutoff):
    """The particle's terms are NaNs, and so is every pixel: not the image of the
    radius that the others have."""
    c, h, b = _group(np.random.default_rng(5), n, basis, "uniform", 0.05)
    h[n // 2] = np.nan
    assert np.isnan(render_direct([(c, h, b)], (1.0, 1.0), cutoff, U, V, (2 * cutoff[0], 2 * cutoff[1]))).all()

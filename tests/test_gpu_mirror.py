"""The tensor form's mirrored elements: half of the row lattice is computed and
the other half comes from the same accumulators (conj(A) B beside A B).  Every
plane where the two halves meet is compared with the FP64 oracle by itself --
a = 0, -1 and -Kx/2, b = 0, -1 and -Ky/2, c = 0 and the Nyquist plane -- for
pure phases (folded and not), h-binned groups and Gaussian groups (axis-
exchanged and not), at particle counts around the 64-particle stage."""
import numpy as np
import pytest

import oracle as O
from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import spectrum_and_views

pytestmark = pytest.mark.gpu

# the tensor form's tolerance on spectra (rel-L2), here on every plane alone:
# the weights are N(0, 1), so no plane's norm is far below the others'
SPEC_TOL = 1e-5

KINDS = {
    "pure": (M.WENDLAND_D3_C2, lambda rng, n: None),
    "uniform": (M.SPH, lambda rng, n: np.full(n, 0.02, np.float32)),
    "binned": (M.WENDLAND_D3_C2, lambda rng, n: rng.uniform(0.004, 0.02, n).astype(np.float32)),
    "gauss": (M.GAUSSIAN_DECAYING, lambda rng, n: rng.uniform(0.002, 0.02, n).astype(np.float32)),
}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("grid", [(32, 32, 32), (48, 64, 32), (64, 48, 96), (64, 128, 32)])
@pytest.mark.parametrize("n", [2, 63, 65, 1029])
def test_mirrored_planes_match_fp64(kind, grid, n):
    rng = np.random.default_rng(n)
    basis, radii = KINDS[kind]
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32)),
               radii(rng, n), basis)]
    spec, _ = spectrum_and_views(groups, grid, 1.0, (1.0, 1.0), (16, 16), (32, 32), None, M.FORM_TENSOR)
    ref = O.spectrum_grid(groups, 1.0, grid)
    assert O.rel_l2(spec, ref) < SPEC_TOL
    hx, hy = grid[0] // 2, grid[1] // 2
    for i in (0, hx - 1, hx, hx + 1):
        assert O.rel_l2(spec[i], ref[i]) < SPEC_TOL, ("a", i - hx)
    for j in (0, hy - 1, hy, hy + 1):
        assert O.rel_l2(spec[:, j], ref[:, j]) < SPEC_TOL, ("b", j - hy)
    for l in (0, 1, grid[2] // 2 - 1, grid[2] // 2):
        assert O.rel_l2(spec[:, :, l], ref[:, :, l]) < SPEC_TOL, ("c", l)
    assert O.rel_l2(spec[:hx, 0], ref[:hx, 0]) < SPEC_TOL  # the Gaussians' face

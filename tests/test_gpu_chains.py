"""What the tensor form adds back for its accumulator's truncation is no more
than truncation can take away.  The sets leave most K steps of a chain without
weight, or have their whole weight at a chain's end, so that little or nothing is
truncated: the coherent part of the error, <error, exact> / <exact, exact>, then
stays below the most that a chain's steps can lose (4.9e-7 of the total per 64
particles) times the share of its steps that count, plus 1e-7 for what is not
the chain's (the dropped product of the operands' low halves, the FP32 slots)."""
import numpy as np
import pytest

import oracle as O
from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import spectrum_and_views

pytestmark = pytest.mark.gpu

MOST_PER_STAGE, REST = 4.9e-7, 1e-7

# lattice, stages of a chain (64 particles each), basis and radii
KINDS = {
    "pure phases": ((64, 64, 64), 8, M.WENDLAND_D3_C2, lambda rng, n: np.full(n, 0.01, np.float32)),
    "h-binned": ((64, 64, 64), 8, M.WENDLAND_D3_C2, lambda rng, n: rng.uniform(0.004, 0.02, n).astype(np.float32)),
    "gaussians": ((64, 64, 256), 16, M.GAUSSIAN_DECAYING, lambda rng, n: rng.uniform(0.0005, 0.003, n).astype(np.float32)),
}


def _coherent_error(kind, weights):
    grid, _, basis, radii = KINDS[kind]
    rng = np.random.default_rng(11)
    n = len(weights)
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), weights.astype(np.float32)), radii(rng, n), basis)]
    spec, _ = spectrum_and_views(groups, grid, 1.0, (1.0, 1.0), (16, 16), (32, 32), None, M.FORM_TENSOR)
    ijk = np.stack([rng.integers(-(grid[0] // 2), grid[0] // 2, 4096), rng.integers(-(grid[1] // 2), grid[1] // 2, 4096),
                    rng.integers(1, grid[2] // 2, 4096)], axis=1)
    got = spec[ijk[:, 0] + grid[0] // 2, ijk[:, 1] + grid[1] // 2, ijk[:, 2]].astype(np.complex128)
    ref = sum(O.spectrum_points(c, h, b, 1.0, ijk) for c, h, b in groups)
    return np.vdot(ref, got - ref).real / np.vdot(ref, ref).real


@pytest.mark.parametrize("kind", list(KINDS))
def test_sparse_weights(kind):
    """One particle in 256: one K step (16 particles) in 16."""
    w = np.zeros(16384)
    w[::256] = np.random.default_rng(1).standard_normal(64)
    assert abs(_coherent_error(kind, w)) < KINDS[kind][1] / 16 * MOST_PER_STAGE + REST


@pytest.mark.parametrize("kind", ["pure phases", "gaussians"])
def test_runs_without_weight(kind):
    """64 particles of each 512: an eighth of a chain's steps."""
    w = np.random.default_rng(2).standard_normal(16384)
    w[np.arange(16384) % 512 >= 64] = 0.0
    assert abs(_coherent_error(kind, w)) < KINDS[kind][1] / 8 * MOST_PER_STAGE + REST


@pytest.mark.parametrize("kind", ["pure phases", "gaussians"])
def test_one_dominant_weight_at_the_end(kind):
    """The last particle of the last chain outweighs all: nothing follows it."""
    w = np.random.default_rng(3).standard_normal(16384)
    w[-1] = 1e5
    assert abs(_coherent_error(kind, w)) < MOST_PER_STAGE + REST

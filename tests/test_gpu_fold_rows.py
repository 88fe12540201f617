"""The folded plain form of SPH and Wendland groups with radii on 3D lattices:
its threads take the (y, z) rows in the order of their distance from the x axis,
and a split's run of particles ends anywhere.  Every element against the FP64
oracle, on lattices whose rows tie in distance (cubes), lie in few planes, or
fill no block, at particle counts around a tile and a split, with radii up to
where Phi^'s table has its last cell."""
import numpy as np
import pytest

import oracle as O
from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import spectrum_and_views

pytestmark = pytest.mark.gpu

# the suite's tolerance on spectra (rel-L2)
SPEC_TOL = 1e-5


@pytest.mark.parametrize("basis", [M.SPH, M.WENDLAND_D3_C2])
@pytest.mark.parametrize("grid", [(16, 16, 16), (20, 18, 14), (6, 34, 2), (14, 4, 50), (22, 70, 30)])
@pytest.mark.parametrize("n,h", [(1, 0.3), (255, 0.02), (1025, 0.1), (3000, 0.9)])
def test_rows_match_fp64(basis, grid, n, h):
    rng = np.random.default_rng(n)
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32)),
               rng.uniform(0.1 * h, h, n).astype(np.float32), basis)]
    spec, _ = spectrum_and_views(groups, grid, 1.0, (1.0, 1.0), (8, 4), (16, 16), None, M.FORM_PLAIN)
    ref = O.spectrum_grid(groups, 1.0, grid)
    assert O.rel_l2(spec, ref) < SPEC_TOL
    # the axis planes by themselves: a row out of its place shows there
    for a, b in ((spec[:, grid[1] // 2], ref[:, grid[1] // 2]), (spec[:, :, 0], ref[:, :, 0])):
        assert O.rel_l2(a, b) < SPEC_TOL


@pytest.mark.parametrize("cells", [2500, 2700, 2900, 3070, 3100])
def test_tables_around_48_kb(cells):
    """A table between 40 KB and 48 KB leaves the kernel's static shared memory
    no room below the size a block gets without asking for more."""
    rng = np.random.default_rng(cells)
    n, kmax, ds = 300, np.sqrt(3.0) * 8, 0.24 / 15.5
    radii = rng.uniform(0.002, 0.2, n).astype(np.float32)
    radii[0] = (cells - 2.5) * ds / kmax
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32)),
               radii, M.WENDLAND_D3_C2)]
    spec, _ = spectrum_and_views(groups, (16, 16, 16), 1.0, (1.0, 1.0), (8, 4), (16, 16), None, M.FORM_PLAIN)
    assert O.rel_l2(spec, O.spectrum_grid(groups, 1.0, (16, 16, 16))) < SPEC_TOL


@pytest.mark.parametrize("radii", ["none", "varying"])
@pytest.mark.parametrize("grid", [(16, 16, 16), (92, 76, 58)])
@pytest.mark.parametrize("n", [257, 513, 2049, 4178])
def test_splits_down_to_one_tile(grid, n, radii):
    """Grids of few blocks split the particles further, into runs around a tile."""
    rng = np.random.default_rng(n)
    h = rng.uniform(0.01, 0.1, n).astype(np.float32) if radii == "varying" else None
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32)), h,
               M.WENDLAND_D3_C2)]
    spec, _ = spectrum_and_views(groups, grid, 1.0, (1.0, 1.0), (8, 4), (16, 16), None, M.FORM_PLAIN)
    assert O.rel_l2(spec, O.spectrum_grid(groups, 1.0, grid)) < SPEC_TOL


@pytest.mark.parametrize("step", [0.1, 0.3, 1.0 / 3.0])
@pytest.mark.parametrize("grid", [(16, 16, 16), (22, 70, 30), (100, 90, 70)])
def test_rows_at_steps_that_are_no_binary_fractions(grid, step):
    """The squared distances of the rows are not exact there: rows that tie, or
    nearly do, still take each place once."""
    rng = np.random.default_rng(7)
    n = 1025
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32)),
               (rng.uniform(0.01, 0.1, n) / step).astype(np.float32), M.WENDLAND_D3_C2)]
    spec, _ = spectrum_and_views(groups, grid, step, (step, step), (8, 4), (16, 16), None, M.FORM_PLAIN)
    ref = O.spectrum_grid(groups, float(np.float32(step)), grid)
    assert O.rel_l2(spec, ref) < SPEC_TOL
    worst = np.abs(spec - ref).reshape(-1).max() / np.abs(ref).reshape(-1).max()
    assert worst < 10 * SPEC_TOL  # no row out of its place, not one element

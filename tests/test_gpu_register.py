"""Registration statistics taken on the device (groups of 8192 terms and more)
and on the host (smaller ones): the weight and radius extremes and the histogram
of the radii decide the weight scales, the h-bins and the route of a group, so a
wrong one shows as a wrong spectrum or an error."""
import numpy as np
import pytest

import oracle as O
from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import spectrum_and_views

pytestmark = pytest.mark.gpu

# the suite's tolerance on spectra (rel-L2)
SPEC_TOL = 1e-5


@pytest.mark.parametrize("n", [8191, 8192, 8193, 30011])
@pytest.mark.parametrize("case", ["spread", "one heavy", "one wide", "zero radius", "all alike", "some negative"])
def test_statistics_match_fp64(n, case):
    rng = np.random.default_rng(n)
    weights = rng.standard_normal(n).astype(np.float32)
    radii = np.exp(rng.uniform(np.log(0.002), np.log(0.05), n)).astype(np.float32)
    if case == "one heavy":
        weights[n - 1] = -300.0
    elif case == "one wide":
        radii[n - 1] = 0.4
    elif case == "zero radius":
        radii[n // 2] = 0.0
    elif case == "all alike":
        radii[:] = np.float32(0.013)
    elif case == "some negative":
        weights[::3] = 0.0
        radii[::3] = -radii[::3]
    groups = [(constraints(rng.random((n, 3), dtype=np.float32), weights), radii, M.WENDLAND_D3_C2)]
    spec, _ = spectrum_and_views(groups, (32, 32, 32), 1.0, (1.0, 1.0), (16, 16), (32, 32), None, M.FORM_AUTO)
    assert O.rel_l2(spec, O.spectrum_grid(groups, 1.0, (32, 32, 32))) < SPEC_TOL


@pytest.mark.parametrize("n", [8191, 8192])
def test_groups_before_a_refused_one_keep_their_statistics(n):
    """The tensor form needs a group's largest |weight|: it takes the first
    group, registered before the second one is refused."""
    rng = np.random.default_rng(n)
    cons = constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32))
    both, first = M.Dataset([(cons, None, M.WENDLAND_D3_C2)] * 2), M.Dataset([(cons, None, M.WENDLAND_D3_C2)])
    both.group(1).number_of_terms = -1
    cfg = M.Config(cutoff=(8, 8), samples=(16, 16), block_length=64)
    with pytest.raises(M.VisError):
        cfg.register(both)
    g, r = first.group(0), both.group(0)
    g.d_constraints, g.d_radii, g.d_number_of_terms = r.d_constraints, r.d_radii, r.d_number_of_terms
    sp = M.Spectrum((32, 32, 32))
    cfg.enable_timing(True)
    sp.compute(cfg, first, M.FORM_TENSOR)
    cfg.synchronize()
    assert cfg.kernel_time(3)[1] > 0  # launches of the tensor kernel
    sp.close()
    cfg.close()

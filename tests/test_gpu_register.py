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


def test_a_new_config_registers_without_mapping_memory():
    """Registered blocks and the statistics' scratch come from the library's
    pool, which keeps what an earlier config gave back: registering the same
    sizes again maps none."""
    import torch

    rng = np.random.default_rng(3)
    n = 8192
    cons = constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32))
    radii = rng.uniform(0.01, 0.05, n).astype(np.float32)

    def mapped():
        cfgs = [M.Config(cutoff=(8, 8), samples=(16, 16), block_length=64) for _ in range(8)]
        sets = [M.Dataset([(cons, radii, M.WENDLAND_D3_C2)]) for _ in cfgs]
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        for cfg, ds in zip(cfgs, sets):
            cfg.register(ds)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        for cfg, ds in zip(cfgs, sets):
            cfg.unregister(ds)
            cfg.close()
        return used

    mapped()
    assert mapped() == 0


@pytest.mark.parametrize("what", ["weight", "first radius", "radius", "infinite radius", "infinite weight"])
def test_host_and_device_statistics_agree_on_nans_and_infinities(what):
    """A set of 8191 terms (host) and the same with one of weight zero more
    (device) take the same route: the same elements are no numbers, or both are
    refused alike."""
    rng = np.random.default_rng(11)
    n = 8192
    weights = rng.standard_normal(n).astype(np.float32)
    radii = np.exp(rng.uniform(np.log(0.01), np.log(0.05), n)).astype(np.float32)
    weights[n - 1] = 0.0
    {"weight": weights, "first radius": radii, "radius": radii, "infinite radius": radii, "infinite weight": weights}[what][
        0 if what == "first radius" else 4000] = np.inf if "infinite" in what else np.nan
    points = rng.random((n, 3), dtype=np.float32)

    def outcome(count):
        cons = constraints(points[:count], weights[:count])
        try:
            spec, images = spectrum_and_views([(cons, radii[:count], M.WENDLAND_D3_C2)], (32, 32, 32), 1.0, (1.0, 1.0),
                                              (16, 16), (32, 32), [((1, 0, 0), (0, 1, 0))], M.FORM_AUTO)
            return np.isfinite(spec), np.isfinite(images)
        except M.VisError as e:
            return str(e)

    host, device = outcome(n - 1), outcome(n)
    if isinstance(host, str) or isinstance(device, str):
        assert host == device
    else:
        assert all(np.array_equal(h, d) for h, d in zip(host, device))

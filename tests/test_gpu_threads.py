"""Host threads with a config each: calls whose tables of Phi^ take different
amounts of shared memory run beside each other, and give what they give alone."""
import threading

import numpy as np
import pytest

from libmeshlessvis_b200 import meshless as M
from libmeshlessvis_b200.workloads import constraints

from util import to_dataset

pytestmark = pytest.mark.gpu


def _set(seed, cells, smax):
    """Radii whose table has `cells` cells (of 0.24 / 15.5) up to |k| = smax."""
    rng = np.random.default_rng(seed)
    n = 300
    h = rng.uniform(0.002, 0.02, n).astype(np.float32)
    h[0] = (cells - 2.5) * (0.24 / 15.5) / smax
    return [(constraints(rng.random((n, 3), dtype=np.float32), rng.standard_normal(n).astype(np.float32)), h,
             M.WENDLAND_D3_C2)]


class _Slices:
    def __init__(self, seed, cells):
        self.cfg = M.Config(cutoff=(16, 16), samples=(32, 32), block_length=64)
        self.ds = to_dataset(_set(seed, cells, np.sqrt(2.0) * 15))
        self.cfg.register(self.ds)

    def call(self):
        self.cfg.render(self.ds)

    def result(self):
        return self.cfg.image()


class _Spectra:
    def __init__(self, seed, cells):
        self.cfg = M.Config(cutoff=(8, 8), samples=(16, 16), block_length=64)
        self.ds = to_dataset(_set(seed, cells, np.sqrt(3.0) * 8))
        self.cfg.register(self.ds)
        self.sp = M.Spectrum((16, 16, 16))

    def call(self):
        self.sp.compute(self.cfg, self.ds, M.FORM_PLAIN)

    def result(self):
        return self.sp.to_host(self.cfg)


@pytest.mark.parametrize("work,small,large", [(_Slices, 1500, 3900), (_Spectra, 2900, 3900)])
def test_tables_of_two_sizes_at_once(work, small, large):
    users = [work(i, cells) for i, cells in enumerate((small, large, small + 50, large - 50))]
    alone = []
    for u in users:
        u.call()
        alone.append(u.result())
    errors = []

    def run(u):
        try:
            for _ in range(3000):
                u.call()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(u,)) for u in users]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for u, ref in zip(users, alone):
        assert np.array_equal(u.result(), ref)

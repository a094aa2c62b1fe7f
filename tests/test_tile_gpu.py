"""The tiled bond kernel (variants 10-13) against the plain one (18): the same bits, with equal and
with varying nodal volumes, with horizons whose records do not fit a tile, at node counts around a
tile's and a slice's edges, and when other kernels broke bonds between its steps."""
import numpy as np
import pytest

from peridem_gb300 import gen
from peridem_gb300.sim import Sim

pytestmark = pytest.mark.gpu
MM = 1e-3


def _impact(n, factor=3.0, vary=False):
    """Two lattice balls of n nodes each at 60 m/s, surfaces 0.2 h apart."""
    rng = np.random.default_rng(n)
    h = 0.1 * MM
    loc = gen.lattice("sphere", 2 * h * np.ceil((n * 0.3) ** (1 / 3) + 1), h)
    loc = loc[np.argsort((loc ** 2).sum(axis=1), kind="stable")[:n]]
    loc = loc[np.lexsort(loc.T[::-1])]
    gap = loc[:, 0].max() - loc[:, 0].min() + 0.4 * h
    parts = [gen.make_particle(loc, h, gen.GLASS, factor, rng, 0.05, (k * gap, 0, 0), vel=(-60.0 * k, 0, 0))
             for k in (0, 1)]
    s = gen.finish(parts, 0.5 * h, 1e-8)
    if vary:
        s.vol *= rng.uniform(0.8, 1.2, len(s.vol))
    return s, gen.base_config(1e-8, 100)


def _same(a, b, P):
    sa, sb = a.state(), b.state()
    for k in sa:
        np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
    for p in range(P):
        np.testing.assert_array_equal(a.connectivity(p), b.connectivity(p))


@pytest.mark.parametrize("n,factor,vary", [(1, 3.0, False), (33, 3.0, False), (127, 3.0, True), (128, 3.0, False),
                                           (129, 3.0, False), (1500, 3.0, True), (1500, 4.0, False),
                                           (4100, 7.5, False)])
def test_tiled_equals_plain(n, factor, vary):
    s, cfg = _impact(n, factor, vary)
    a = Sim(s, cfg, "fp32c")
    a.tune(graphs=1)
    a.set_variant(18)
    a.step(24)
    full = [len(s.particle_conn(p)) for p in range(2)]
    if n >= 127 and factor == 3.0:
        assert any(len(a.connectivity(p)) < full[p] for p in range(2))  # bonds broke
    for v in (10, 11, 12, 13):
        b = Sim(s, cfg, "fp32c")
        b.tune(graphs=1)
        b.set_variant(v)
        b.step(24)
        _same(a, b, 2)
        b.close()


def test_other_kernels_between_tiled_steps():
    s, cfg = _impact(900)
    a, b = Sim(s, cfg, "fp32c"), Sim(s, cfg, "fp32c")
    a.tune(graphs=1)
    a.set_variant(18)
    b.set_variant(10)
    for mode, v in ((1, 10), (1, 18), (1, 10), (3, 10), (1, 11), (0, 12)):
        b.tune(graphs=mode)
        b.set_variant(v)
        b.step(8)
        a.step(8)
        _same(a, b, 2)
    b.snapshot()
    b.step(8)
    b.restore()
    b.step(4)
    a.step(4)
    _same(a, b, 2)

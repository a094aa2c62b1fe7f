"""The tiled bond kernel (variants 10-13) against the plain one (18): the same bits, with equal and
with varying nodal volumes, with horizons whose records do not fit a tile, at node counts around a
tile's and a slice's edges, and when other kernels broke bonds between its steps."""
import mmap

import numpy as np
import pytest

from peridem_gb300 import gen
from peridem_gb300._capi import lib, ptr
from peridem_gb300.sim import Batch, Sim, estimate_bytes
from tests import cases

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


@pytest.mark.parametrize("name", ["impact_free", "toggles"])
def test_every_variant_in_the_step_graph(name):
    """Each bond-kernel variant stepping in the step graph (a small handle's default, the persistent step,
    has a bond loop of its own): the same bits as variant 18 and as the default."""
    s, cfg = cases.CASES[name]()

    def run(v):
        a = Sim(s, cfg, "fp32c")
        if v is not None:
            a.tune(graphs=1)
            a.set_variant(v)
            assert a.graph_mode() == 1
        a.step(25)
        return a

    ref = run(18)
    _same(ref, run(None), s.n_particles)
    for v in range(lib().pd_num_variants()):
        _same(ref, run(v), s.n_particles)


def test_default_path_of_a_large_handle():
    """Just above the size from which a handle has tiles when it is created: a packing in contact with its
    walls and a breaking impact in one handle, stepped as it comes, as larger handles step (conditional
    graph, variant 10) and in the persistent launch, against variant 18 -- with a member that finishes
    on the way. The memory estimate includes the tiles, and state reads give the same into pages in
    use and untouched ones."""
    items = [gen.crush_contact(count=24), gen.two_sphere(R=1e-3, v=60.0, gap=0.1, seed=2)]
    setups, cfgs = [s for s, _ in items], [c for _, c in items]
    est = estimate_bytes(setups, "fp32c")

    def run(graphs, variant):
        b = Batch(setups, cfgs, "fp32c")
        assert 163840 <= b.N < 1 << 18 and b.device_bytes() == est
        if graphs:
            b.tune(graphs=graphs)
        else:
            assert b.graph_mode() == 1
        if variant:
            b.set_variant(variant)
        b.step(25)
        mid = b.state()
        b.finish(1)
        b.step(10)
        return b, mid

    ref, want = run(1, 18)
    n0 = [len(s.conn) for s in setups]
    for graphs, variant in ((0, 0), (2, 10), (3, 0)):
        b, mid = run(graphs, variant)
        for k in want:
            np.testing.assert_array_equal(mid[k], want[k], err_msg=k)
        left = [0, 0]
        for i in (0, 1):
            x, y = b.sim_state(i), ref.sim_state(i)
            for k in x:
                np.testing.assert_array_equal(x[k], y[k], err_msg=f"{i} {k}")
            for p in range(setups[i].n_particles):
                c = b.sim_connectivity(i, p)
                np.testing.assert_array_equal(c, ref.sim_connectivity(i, p))
                left[i] += len(c)
        assert left[1] < n0[1]  # bonds broke
        b.close()
    used = np.full((ref.N, 3), 7.0)
    new = np.frombuffer(mmap.mmap(-1, ref.N * 24), dtype=np.float64).reshape(ref.N, 3)
    for out in (new, used):
        assert lib().pd_get_node_state(ref.h, ptr(out), None, None, None, None) == 0
    np.testing.assert_array_equal(new, used)
    ref.close()


def test_step_bytes_of_the_kernel_in_use():
    s, cfg = _impact(900)
    a = Sim(s, cfg, "fp32c")
    nodes, tiles = 224.0 * s.n_nodes, -(-s.n_nodes // 256)
    a.set_variant(18)
    assert a.step_bytes() == 4.125 * s.n_bonds_directed + nodes
    a.set_variant(10)
    lists = a.step_bytes() - 2.0 * s.n_bonds_directed - nodes
    assert 4 * s.n_nodes <= lists <= 4 * min(3072, s.n_nodes) * tiles


def test_tiles_built_on_a_callers_stream():
    """The tile arrays are allocated when a variant first needs them, in the handle's own stream, and
    built and read on the stream the caller chose meanwhile, beside another handle that does the same."""
    torch = pytest.importorskip("torch")
    s, cfg = _impact(900)
    ref = Sim(s, cfg, "fp32c")
    ref.tune(graphs=1)
    ref.set_variant(18)
    ref.step(16)
    streams = [torch.cuda.Stream() for _ in range(2)]
    sims = [Sim(s, cfg, "fp32c") for _ in streams]
    for a, q in zip(sims, streams):
        a.set_stream(q.cuda_stream)
        a.tune(graphs=1)
        a.step(8, sync=False)
    for a in sims:
        a.set_variant(10)
        a.step(8, sync=False)
    for a in sims:
        a.sync()
        _same(a, ref, 2)
        a.set_stream(None)
        a.close()


@pytest.mark.parametrize("other", ["wide", "bondless"])
def test_default_kernel_of_a_large_handle_by_its_tiles(other):
    """Tiles are the default from 163,840 nodes on unless some tile's records do not fit; tiles without
    bonds do not count. pd_step_bytes tells the kernels apart."""
    h, rng = 0.1 * MM, np.random.default_rng(0)

    def part(n, factor, x):
        loc = gen.lattice("cube", n * h, h)
        return gen.make_particle(loc, h, gen.GLASS, factor, rng, 0.05, (x * h, 0, 0))

    gen.set_bond_builder("gpu")
    try:
        s = gen.finish([part(56, 2.0, 0.0), part(20, 6.0 if other == "wide" else 0.5, 60.0)], 0.5 * h, 1e-8)
    finally:
        gen.set_bond_builder("cpu")
    a = Sim(s, gen.base_config(1e-8, 10), "fp32c")
    plain = 4.125 * s.n_bonds_directed + 224.0 * s.n_nodes
    assert a.step_bytes() == plain if other == "wide" else a.step_bytes() < plain
    b = Sim(s, gen.base_config(1e-8, 10), "fp32c")
    b.tune(graphs=1)
    b.set_variant(12 if other == "wide" else 18)
    a.step(3)
    b.step(3)
    _same(a, b, 2)

"""Appends of a short batch by one block: repeats in both orders, edges already
present, loops, bad ids and a hub that takes many of them, at batch sizes
around a block's warps and around the sizes where the append changes its form.
Counts and lists as one-by-one appends give them, and the state the oracle's."""
import numpy as np
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _batch(g, n, seed):
    rng = np.random.default_rng(seed)
    p = rng.integers(0, g.nv, size=(n, 2))
    p[rng.random(n) < 0.3, 0] = 5
    for i in range(1, n):
        r = rng.random()
        if r < 0.2:
            p[i] = p[rng.integers(0, i)][::-1]
        elif r < 0.3:
            p[i] = G.edge_list(g)[rng.integers(0, g.ne)]
    if n > 2:
        p[n // 2] = (9, 9)
        p[n // 3] = (g.nv, 2)
    return p


def _apply(g, batch):
    """One-by-one appends: the counts and the graph they leave."""
    live = {tuple(x) for x in G.edge_list(g).tolist()}
    n = {"inserted": 0, "duplicates": 0, "invalid": 0}
    for u, v in batch.tolist():
        k = (min(u, v), max(u, v))
        if u == v or k[1] >= g.nv:
            n["invalid"] += 1
        elif k in live:
            n["duplicates"] += 1
        else:
            live.add(k)
            n["inserted"] += 1
    e = np.asarray(sorted(live))
    return n, G.from_edges(g.nv, e[:, 0], e[:, 1])


def _check(dg, f, g, roots, port_lib):
    off, adj = dg.to_csr()
    for v in range(g.nv):
        np.testing.assert_array_equal(np.sort(adj[off[v]:off[v + 1]]), np.sort(g.adj[g.off[v]:g.off[v + 1]]))
    o = port_lib.PortOracle(g.nv, g.off, g.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    o.close()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 130])
def test_short_batches(sbc_lib, port_lib, n):
    g = G.er(150, 400, seed=n)
    roots = G.pick_roots(g.nv, 17, seed=n)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    for step in range(3):  # later batches meet lists that an earlier one sealed
        b = _batch(g, n, 10 * n + step)
        want, g = _apply(g, b)
        st = f.insert(b)
        assert {k: st[k] for k in want} == want
        _check(dg, f, g, roots, port_lib)
    f.close()
    dg.close()


def test_group_batches_around_the_block(sbc_lib, port_lib):
    sizes = [0, 1, 33, 255, 256, 257]
    gs = [G.er(200, 500, seed=s) for s in range(len(sizes))]
    roots = [G.pick_roots(g.nv, 9, seed=1) for g in gs]
    dgs = [native.DeviceGraph(g.nv, g.off, g.adj) for g in gs]
    fs = [native.DeviceForest(d, r) for d, r in zip(dgs, roots)]
    for f in fs:
        f.static_init()
    grp = native.DeviceGroup(fs)
    for step in range(2):
        batches = [_batch(g, n, n + step) for g, n in zip(gs, sizes)]
        grp.insert(batches)
        gs = [_apply(g, b)[1] for g, b in zip(gs, batches)]
        for d, f, g, r in zip(dgs, fs, gs, roots):
            _check(d, f, g, r, port_lib)
    grp.close()
    for d, f in zip(dgs, fs):
        f.close()
        d.close()

"""Removal marks of a deletion call, found a warp per deletion: the same edge
named several times and in both orders, edges that are absent, bad ids, calls
around a warp's width, and lists with an unsorted tail.  Counts as one-by-one
deletions give them, and the state the oracle's."""
import numpy as np
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _check(f, g, roots, port_lib):
    o = port_lib.PortOracle(g.nv, g.off, g.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    o.close()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 70])
@pytest.mark.parametrize("mode", [native.DeviceForest.DELETE_MOVE_DOWN, native.DeviceForest.DELETE_RECOMPUTE])
def test_repeated_and_absent_deletions(sbc_lib, port_lib, n, mode):
    g = G.er(260, 1500, seed=n)
    roots = G.pick_roots(g.nv, 19, seed=n)
    rng = np.random.default_rng(n)
    e = G.edge_list(g)
    some = e[rng.choice(len(e), max(1, n // 2), replace=False)]
    picks = some[rng.integers(0, len(some), n)]  # most of them more than once
    flip = rng.random(n) < 0.5
    picks[flip] = picks[flip][:, ::-1]
    if n > 2:
        picks[n // 2] = (7, 7)
        picks[n // 3] = (3, g.nv)
        picks[n - 1] = G.uniform_insertions(g, 1, seed=n)[0]
    want = {"inserted": 0, "duplicates": 0, "invalid": 0}
    live = {tuple(x) for x in e.tolist()}
    for u, v in picks.tolist():
        k = (min(u, v), max(u, v))
        if u == v or k[1] >= g.nv:
            want["invalid"] += 1
        elif k in live:
            live.remove(k)
            want["inserted"] += 1
        else:
            want["duplicates"] += 1
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.set_delete_mode(mode)
    f.static_init()
    st = f.delete(picks)
    assert {k: st[k] for k in want} == want
    left = np.asarray(sorted(live))
    _check(f, G.from_edges(g.nv, left[:, 0], left[:, 1]), roots, port_lib)
    f.close()
    dg.close()


def test_deletions_from_an_unsorted_tail(sbc_lib, port_lib):
    """A batch that appends more slots to one vertex than one merge takes leaves a tail behind; deletions find
    their slots there and before it."""
    nv = 2600
    g = G.from_edges(nv, np.arange(nv - 1), np.arange(1, nv))
    roots = np.asarray([0, 40, 2000, 2599])
    ins = np.stack([np.full(2300, 5), np.r_[8:2308]], 1)
    dg = native.DeviceGraph(nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    assert f.insert(ins)["inserted"] == len(ins)
    dels = np.asarray([(5, 2307), (2307, 5), (5, 9), (5, 2200), (5, 2306), (5, 2599), (9, 5)])
    st = f.delete(dels)
    assert (st["inserted"], st["duplicates"], st["invalid"]) == (4, 3, 0)
    _check(f, G.delete_edges(G.insert_edges(g, ins), dels), roots, port_lib)
    f.close()
    dg.close()


@pytest.mark.parametrize("nv,m,call", [(300, 900, 5), (300, 900, 40), (2000, 5000, 16)])
def test_level2_masks_follow_deletions(sbc_lib, port_lib, nv, m, call):
    """Deletions around the roots' neighbours (edges of a root, of its neighbours, between two of them, and others),
    many in one call, with roots of few and of more than 32 neighbours; then insertions that rely on the masks."""
    rng = np.random.default_rng(nv + call)
    g = G.er(nv, m, seed=call)
    hub = np.stack([np.full(50, 4), rng.choice(np.arange(5, nv), 50, replace=False)], 1)
    g = G.insert_edges(g, hub)
    roots = np.asarray(sorted({4, *rng.choice(np.arange(5, nv), 11, replace=False).tolist()}))
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.set_delete_mode(native.DeviceForest.DELETE_MOVE_DOWN)
    f.static_init()
    for step in range(3):
        e = G.edge_list(g)
        near = np.isin(e, roots).any(1)
        nb = np.unique(e[near])
        second = np.isin(e, nb).any(1) & ~near
        pick = np.concatenate([rng.permutation(e[near])[:call // 5 + 1], rng.permutation(e[second])[:call],
                               rng.permutation(e)[:call // 3 + 1]])
        pick = rng.permutation(np.unique(pick, axis=0))[:call]
        assert f.delete(pick)["inserted"] == len(pick)
        g = G.delete_edges(g, pick)
        _check(f, g, roots, port_lib)
        ins = G.uniform_insertions(g, 8, seed=step)
        assert f.insert(ins)["inserted"] == 8
        g = G.insert_edges(g, ins)
        _check(f, g, roots, port_lib)
    f.close()
    dg.close()

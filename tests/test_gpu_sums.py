"""Static init's dependencies against Brandes in long double: long lists are
summed in parallel chains, whichever side their level pair is walked from."""
import numpy as np
import pytest

from _util import INF32
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _delta(g, root):
    """Levels, dependencies in long double, and the number of levels."""
    src = np.repeat(np.arange(g.nv), np.diff(g.off))
    dist = np.full(g.nv, INF32)
    sigma = np.zeros(g.nv, dtype=np.longdouble)
    delta = np.zeros(g.nv, dtype=np.longdouble)
    dist[root], sigma[root], lv = 0, 1, 0
    steps = []
    while True:
        e = (dist[src] == lv) & (dist[g.adj] == INF32)
        dist[g.adj[e]] = lv + 1
        e = (dist[src] == lv) & (dist[g.adj] == lv + 1)
        if not e.any():
            break
        np.add.at(sigma, g.adj[e], sigma[src[e]])
        steps.append(e)
        lv += 1
    for e in reversed(steps):
        x, k = src[e], g.adj[e]
        sums = np.zeros(g.nv, dtype=np.longdouble)
        np.add.at(sums, x, (delta[k] + 1) / sigma[k])
        delta += sigma * sums
    return dist, delta, len(steps)


def _bipartite(hubs, leaves, per, seed):
    """Every hub joined to `per` of the leaves (all of them: 0)."""
    if per == 0:
        return G.from_edges(hubs + leaves, np.repeat(np.arange(hubs), leaves), np.tile(np.arange(hubs, hubs + leaves), hubs))
    rng = np.random.default_rng(seed)
    v = np.concatenate([rng.choice(leaves, per, replace=False) for _ in range(hubs)]) + hubs
    return G.from_edges(hubs + leaves, np.repeat(np.arange(hubs), per), v)


# whole rows in shared memory and bitmaps alone; few long lists (summed in segments) and more of them than a walk lists
@pytest.mark.parametrize("hubs,leaves,per", [(1, 5000, 0), (3, 7000, 0), (5, 60000, 0), (100, 3000, 200),
                                             (1500, 9000, 150), (1500, 9000, 100)])
def test_dependencies_of_hubs(sbc_lib, hubs, leaves, per):
    g = _bipartite(hubs, leaves, per, seed=hubs)
    roots = np.array([0, hubs, hubs + leaves // 2, hubs + leaves - 1])
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    # the longest chain of additions of a sum: a push's (fewer than 128 neighbours here), or a lane's share of a segment
    # of 2,048, the warp's tree and the list's segments; beside it a level takes fewer than 8 roundings, and each level's
    # error is at most that of the levels below and its own
    chain = max(128, 2048 // 32 + 5 + -(-int(g.degrees().max()) // 2048))
    dist = f.dist()
    for i, r in enumerate(roots):
        lv, want, levels = _delta(g, int(r))
        assert np.array_equal(dist[i], lv)
        got = f.delta(i, 1)[0]
        ok = want != 0
        assert np.all(got[~ok] == 0)
        err = np.abs((got[ok] - want[ok]) / want[ok])
        assert float(err.max()) <= 1.01 * levels * (chain + 8) * 2.0 ** -53
    f.close()
    dg.close()

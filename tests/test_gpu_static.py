"""Static init where its kernel changes form: the working set of a root in
shared memory, only the bitmaps there, one of them or none (by vertex count),
vertices scanned by a thread, 4 or 16 lanes, a warp or the CTA (by degree), levels
walked from above or below, and adjacencies that are not symmetric.  dist and
sigma bit-exact against the oracle, BC within the 1e-9 of the parity tests."""
import numpy as np
import pytest

from _util import INF32, assert_bc, assert_levels, assert_sigma, bc_err
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _mixed(nv, seed):
    """A hub over half of the vertices (20,000 at most), a path hanging off it, random edges among the hub's
    neighbours, a small separate clique, and isolated vertices."""
    rng = np.random.default_rng(seed)
    leaves = max(1, min(nv // 2, 20000))
    path = min(70, nv // 8)
    u = [np.zeros(leaves, np.int64)]
    v = [np.arange(1, leaves + 1)]
    u.append(np.arange(leaves, leaves + path))
    v.append(np.arange(leaves + 1, leaves + path + 1))
    m = 3 * leaves
    u.append(rng.integers(1, leaves + 1, m))
    v.append(rng.integers(1, min(nv - 1, 2 * leaves) + 1, m))
    if nv > 40:
        c = np.arange(nv - 6, nv)
        a, b = np.meshgrid(c, c)
        u.append(a.ravel())
        v.append(b.ravel())
    g = G.from_edges(nv, np.minimum(np.concatenate(u), nv - 1), np.minimum(np.concatenate(v), nv - 1))
    roots = sorted({0, min(1, nv - 1), leaves, min(leaves + path, nv - 1), nv // 2, int(nv * 0.9), nv - 1})
    return g, np.asarray(roots, dtype=np.int64)


# around the largest graph whose rows fit in shared memory (about 7,860 vertices), and the sizes of which two
# bitmaps (about 0.89 million) or one (1.77 million) do
@pytest.mark.parametrize("nv", [2, 31, 33, 200, 1025, 4100, 7800, 7900, 45001, 300007, 1000003, 1800001])
def test_static_at_every_size_class(sbc_lib, port_lib, nv):
    g, roots = _mixed(nv, seed=nv)
    if nv > 500000:
        roots = roots[:4]
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    f.static_init()  # scratch left clean by the first
    o = port_lib.PortOracle(g.nv, g.off, g.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    d = f.dist()
    h = np.stack([np.bincount(np.minimum(row[row != INF32], 63), minlength=64) for row in d])
    assert np.array_equal(f.level_hist(), h)
    for r in range(len(roots)):
        for lv in range(2, 16):
            ros = f.roster(r, lv)
            want = np.flatnonzero(d[r] == lv)
            assert (ros is None) == (want.size > 256)
            assert ros is None or np.array_equal(np.sort(ros), want)
    o.close()
    # the rows derived with the levels serve the updates
    ins = G.uniform_insertions(g, 6, seed=nv) if nv > 33 else np.zeros((0, 2), np.int64)
    f.insert(ins)
    o = port_lib.PortOracle(*_csr(G.insert_edges(g, ins)), roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    o.close()
    f.close()
    dg.close()


def _csr(g):
    return g.nv, g.off, g.adj


def _directed(nv, off, adj, root):
    """Levels, path counts and dependencies along out-edges."""
    dist, sigma, delta = np.full(nv, INF32), np.zeros(nv, dtype=np.int64), np.zeros(nv)
    dist[root], sigma[root] = 0, 1
    levels = [[root]]
    while levels[-1]:
        nxt = []
        for x in levels[-1]:
            for k in adj[off[x]:off[x + 1]]:
                if dist[k] == INF32:
                    dist[k] = dist[x] + 1
                    nxt.append(k)
                if dist[k] == dist[x] + 1:
                    sigma[k] += sigma[x]
        levels.append(nxt)
    for lv in reversed(levels):
        for x in lv:
            c = [k for k in adj[off[x]:off[x + 1]] if dist[k] == dist[x] + 1]
            delta[x] = sigma[x] * sum((delta[k] + 1) / sigma[k] for k in c)
    return dist, sigma, delta


@pytest.mark.parametrize("nv,k", [(60, 60), (9000, 5)])
def test_static_follows_stored_directions(sbc_lib, nv, k):
    """An adjacency stored in one direction only is walked along its stored slots; a directed insertion and its
    removal switch between the two forms."""
    rng = np.random.default_rng(nv)
    src = np.repeat(np.arange(nv), 3)
    dst = rng.integers(0, nv, src.size)
    keep = src < nv - 4  # the last vertices have no out-edges
    deg = np.bincount(src[keep], minlength=nv)
    off = np.concatenate([[0], np.cumsum(deg)])
    adj = np.concatenate([np.sort(dst[keep][off[v]:off[v + 1]]) for v in range(nv)])
    roots = np.sort(rng.choice(nv, k, replace=False))
    dg = native.DeviceGraph(nv, off, adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    d, s, dl = f.dist(), f.sigma(), f.delta()
    for i, r in enumerate(roots):
        wd, ws, wl = _directed(nv, off, adj, int(r))
        assert np.array_equal(d[i], wd)
        assert np.array_equal(s[i], ws)
        assert bc_err(dl[i], wl) <= 1e-9
    f.close()
    dg.close()
    g = G.er(nv, 4 * nv, seed=nv)
    dg = native.DeviceGraph(nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    want = f.dist(), f.sigma()
    u = int(roots[0])
    v = int(np.flatnonzero(want[0][0] > 1)[0])
    assert dg.insert_directed(u, v) == 1
    f.static_init()
    off, adj = dg.to_csr()
    wd, ws, _ = _directed(nv, off, adj, u)
    assert np.array_equal(f.dist(0, 1)[0], wd) and np.array_equal(f.sigma(0, 1)[0], ws)
    assert dg.remove_directed(u, v) == 1
    f.static_init()
    assert np.array_equal(f.dist(), want[0]) and np.array_equal(f.sigma(), want[1])
    f.close()
    dg.close()

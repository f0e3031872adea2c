"""Deletion calls large enough that several of their edges share endpoints:
every list afterwards holds the graph's edges, each once, whichever of a
vertex's blocks came to it first."""
import numpy as np
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,batch,steps", [(300, 2, 3), (300, 600, 3), (20000, 2000, 6), (20000, 10000, 3)])
def test_lists_after_large_deletions(sbc_lib, port_lib, nv, batch, steps):
    g = G.er(nv, 5 * nv, seed=1)
    roots = G.pick_roots(nv, 6, seed=batch)
    ins = G.uniform_insertions(g, 3 * batch, seed=batch).reshape(3, batch, 2)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    assert f.insert(ins[0])["inserted"] == batch
    for step in range(steps):
        assert f.insert(ins[(step + 1) % 3])["inserted"] == batch
        assert f.delete(ins[step % 3])["inserted"] == batch
        now = G.insert_edges(g, ins[(step + 1) % 3])
        off, adj = dg.to_csr()
        np.testing.assert_array_equal(np.diff(off), np.diff(now.off))
        src = np.repeat(np.arange(nv), np.diff(off))
        np.testing.assert_array_equal(np.sort(src * nv + adj), now.edge_keys())
    o = port_lib.PortOracle(now.nv, now.off, now.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    o.close()
    f.close()
    dg.close()

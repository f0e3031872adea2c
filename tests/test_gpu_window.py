"""A window of edges that come and go: the host's degree bounds follow the
removals, so the adjacency is re-packed once at most, and every call's
statistics and state are those of the graph at that point."""
import numpy as np
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 5, 64, 70])
def test_window_of_edges(sbc_lib, port_lib, batch):
    g = G.er(400, 1600, seed=batch)
    roots = G.pick_roots(g.nv, 40, seed=batch)
    ins = G.uniform_insertions(g, 3 * batch, seed=batch).reshape(3, batch, 2)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    assert f.insert(ins[0])["inserted"] == batch
    for step in range(12):
        new, old = ins[(step + 1) % 3], ins[step % 3]
        st = f.insert(np.concatenate([new, [(3, 3)], old[:1]]))
        assert (st["inserted"], st["duplicates"], st["invalid"]) == (batch, 1, 1)
        st = f.delete(np.concatenate([old, [(-1, 2)], old[:1]]))
        assert (st["inserted"], st["duplicates"], st["invalid"]) == (batch, 1, 1)
    # a step inserts `batch` edges and one duplicate, which the bounds count
    assert dg.repacks() <= 4
    now = G.insert_edges(g, ins[12 % 3])
    o = port_lib.PortOracle(now.nv, now.off, now.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    off, adj = dg.to_csr()
    assert sorted(zip(np.repeat(np.arange(g.nv), np.diff(off)).tolist(), adj.tolist())) == \
        sorted(zip(np.repeat(np.arange(g.nv), np.diff(now.off)).tolist(), now.adj.tolist()))
    o.close()
    f.close()
    dg.close()

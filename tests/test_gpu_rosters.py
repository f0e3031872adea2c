"""Vertices that move down in one call and up again in the next: no roster names
one twice, and the state is that of a static init."""
import numpy as np
import pytest

from _util import assert_bc
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _hub(nv, seed):
    """A hub over most vertices, random edges, and a few short tails."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([np.zeros(nv - 20, np.int64), rng.integers(0, nv, nv // 2), np.arange(nv - 20, nv - 1)])
    v = np.concatenate([np.arange(1, nv - 19), rng.integers(0, nv, nv // 2), np.arange(nv - 19, nv)])
    return G.from_edges(nv, u, v)


@pytest.mark.parametrize("one_by_one", [False, True])
@pytest.mark.parametrize("nv,batch", [(150, 50), (400, 30)])
def test_down_and_up_again(sbc_lib, nv, batch, one_by_one):
    rng = np.random.default_rng(nv)
    g = _hub(nv, nv)
    roots = np.arange(nv)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.set_delete_mode(f.DELETE_MOVE_DOWN)
    f.static_init()
    for step in range(4):
        e = G.edge_list(g)
        gone = e[rng.choice(len(e), batch, replace=False)]
        if one_by_one:
            for u, v in gone:
                assert dg.remove_directed(int(u), int(v)) == 1 and dg.remove_directed(int(v), int(u)) == 1
                f.update_deleted(int(u), int(v))
        else:
            assert f.delete(gone)["inserted"] == batch
        g = G.delete_edges(g, gone)
        # half of them come back, and others
        new = np.concatenate([gone[: batch // 2], G.uniform_insertions(g, batch, seed=step)])
        f.insert(new)
        g = G.insert_edges(g, new)
        g2 = native.DeviceGraph(g.nv, g.off, g.adj)
        fresh = native.DeviceForest(g2, roots)
        fresh.static_init()
        d = fresh.dist()
        assert np.array_equal(f.dist(), d)
        assert np.array_equal(f.sigma(), fresh.sigma())
        for r in range(nv):
            for lv in range(2, 16):
                ros = f.roster(r, lv)
                if ros is not None:
                    assert np.array_equal(np.sort(ros), np.flatnonzero(d[r] == lv))
        assert_bc(f.bc(), fresh.bc())
        for r in range(nv):
            assert_bc(f.delta(r, 1)[0], fresh.delta(r, 1)[0])
        fresh.close()
        g2.close()
    f.close()
    dg.close()

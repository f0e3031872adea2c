"""Static init of deep trees and of levels that are short beside the graph:
paths, narrow grids, trees, lists of up to four neighbours beside longer ones,
levels around the number of threads.  dist and sigma bit-exact against the
oracle, BC within the 1e-9 of the parity tests."""
import numpy as np
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _grid(a, b):
    i = np.arange(a * b).reshape(a, b)
    return np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()]), np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])


def _tree(levels, fan=2):
    nv = (fan ** levels - 1) // (fan - 1)
    v = np.arange(1, nv)
    return nv, (v - 1) // fan, v


def _graph(name):
    if name.startswith("path"):
        nv = int(name[4:])
        return nv, np.arange(nv - 1), np.arange(1, nv)
    if name.startswith("grid"):
        a, b = map(int, name[4:].split("x"))
        return a * b, *_grid(a, b)
    if name == "tree":      # levels of 1,024 and 2,048 listed as they come, longer ones in vertex order
        return _tree(17)
    if name == "fan5":      # inner vertices of six neighbours, leaves of one
        return _tree(7, 5)
    # a path whose every tenth vertex carries 9 leaves, and a chord here and there
    nv = 12000
    spine = np.arange(0, nv // 2)
    leaves = np.arange(nv // 2, nv)
    at = (np.arange(leaves.size) // 9) * 10 % spine.size
    return nv, np.concatenate([spine[:-1], at, [3, 700]]), np.concatenate([spine[1:], leaves, [900, 1200]])


@pytest.mark.parametrize("name", ["path300", "path9000", "grid6x300", "grid6x1500", "tree", "fan5", "comb"])
def test_deep_and_short_levels(sbc_lib, port_lib, name):
    nv, u, v = _graph(name)
    g = G.from_edges(nv, u, v)
    roots = np.unique([0, 1, nv // 3, nv // 2, nv - 1])
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    f.static_init()  # scratch left clean by the first
    o = port_lib.PortOracle(g.nv, g.off, g.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    for r in range(len(roots)):
        assert_bc(f.delta(r, 1)[0], o.delta()[r])
    o.close()
    f.close()
    dg.close()


@pytest.mark.parametrize("nv", [40, 63, 64, 65, 66, 67, 300, 9000])
def test_scanned_slots_of_a_path(sbc_lib, nv):
    """From one end of a path every level is one vertex: all slots are read on the way down, and on the way up those
    of every vertex but the last, or one fewer where the last two levels are walked from the last."""
    g = G.from_edges(nv, np.arange(nv - 1), np.arange(1, nv))
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, [0])
    f.counters()
    f.static_init()
    down = 2 * (nv - 1)
    assert down + down - 2 <= f.counters()["scanned"] <= down + down - 1
    f.close()
    dg.close()

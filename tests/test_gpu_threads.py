"""Calls on different graphs from different host threads at the same time."""
import threading

import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


# the graphs of a set run one kernel with different amounts of shared memory: whole rows, bitmaps
@pytest.mark.parametrize("sizes,reps", [((7500, 2100, 6000, 3100, 7000, 4100), 2000), ((700000, 300000, 500000), 40)])
def test_static_init_beside_other_graphs(sbc_lib, port_lib, sizes, reps):
    gs = [G.er(nv, nv // 2, seed=nv) for nv in sizes]
    roots = [G.pick_roots(g.nv, 2, seed=1) for g in gs]
    dgs = [native.DeviceGraph(g.nv, g.off, g.adj) for g in gs]
    fs = [native.DeviceForest(d, r) for d, r in zip(dgs, roots)]
    errors = []

    def work(f):
        try:
            for i in range(reps):
                f.static_init(sync=i % 20 == 19)
        except native.SbcError as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(f,)) for f in fs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    for g, f, r in zip(gs, fs, roots):
        o = port_lib.PortOracle(g.nv, g.off, g.adj, r, nthreads=2)
        o.static()
        assert_levels(f.level64(), o.level())
        assert_sigma(f.sigma(), o.sigma(), o.level())
        assert_bc(f.bc(), o.bc())
        o.close()
    for d, f in zip(dgs, fs):
        f.close()
        d.close()


def test_graphs_built_beside_work_on_the_default_stream(sbc_lib):
    """A graph's arrays are filled on its own stream, whatever another thread has queued on the default one."""
    torch = pytest.importorskip("torch")
    g = G.er(3000, 30000, seed=1)
    x = torch.randn(2048, 2048, device="cuda")
    stop = threading.Event()

    def busy():
        while not stop.is_set():
            for _ in range(20):
                torch.mm(x, x)
            torch.cuda.default_stream().synchronize()

    t = threading.Thread(target=busy)
    t.start()
    try:
        for _ in range(60):
            dg = native.DeviceGraph(g.nv, g.off, g.adj)
            off, adj = dg.to_csr()
            dg.close()
            assert (off == g.off).all() and (adj == g.adj).all()
    finally:
        stop.set()
        t.join()

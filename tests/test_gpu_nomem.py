"""A batch too large to be staged in the memory that is left is refused, and the
graph and the forest work on."""
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def test_staging_that_does_not_fit(sbc_lib, port_lib):
    torch = pytest.importorskip("torch")
    g = G.er(300, 1200, seed=1)
    roots = G.pick_roots(g.nv, 30, seed=1)
    ins = G.uniform_insertions(g, 20, seed=1)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    f.insert(ins[:10])
    n = 100_000_000  # 2 GB of staging; were it staged, all of it loops, which are refused one by one
    same = torch.zeros(n, dtype=torch.int32, device="cuda")
    free, _ = torch.cuda.mem_get_info()
    rest = torch.empty(free - (512 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(native.SbcError):
        f.insert_device(n, same.data_ptr(), same.data_ptr())
    f.sync()
    assert f.insert(ins[10:])["inserted"] == 10
    del rest, same
    torch.cuda.empty_cache()
    now = G.insert_edges(g, ins)
    o = port_lib.PortOracle(now.nv, now.off, now.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    o.close()
    f.close()
    dg.close()

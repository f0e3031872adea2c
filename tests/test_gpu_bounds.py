"""The host's degree bounds when device batches and deletions mix: a host batch
finds room (or re-packs) whatever device batches took from the slack before
it, and a device window that reserves each batch re-packs once at most."""
import numpy as np
import pytest

from _util import assert_bc, assert_levels, assert_sigma
from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _start(nv, seed):
    torch = pytest.importorskip("torch")
    g = G.er(nv, 3 * nv, seed=seed)
    roots = G.pick_roots(g.nv, 30, seed=seed)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, roots)
    f.static_init()
    hub = int(np.argmax(g.degrees()))
    near = set(g.adj[g.off[hub]:g.off[hub + 1]].tolist()) | {hub}
    fresh = np.array([(hub, x) for x in range(g.nv) if x not in near], dtype=np.int64)

    def device(pairs):
        d = torch.tensor(np.asarray(pairs), dtype=torch.int32, device="cuda")
        u, v = d[:, 0].contiguous(), d[:, 1].contiguous()
        torch.cuda.synchronize()  # they are made on another stream than the forest's
        f.insert_device(len(d), u.data_ptr(), v.data_ptr())
        f.sync()

    return g, roots, dg, f, hub, near - {hub}, fresh, device


def _check(port_lib, g, roots, dg, f):
    off, adj = dg.to_csr()
    src = np.repeat(np.arange(g.nv), np.diff(off))
    np.testing.assert_array_equal(np.sort(src * g.nv + adj), g.edge_keys())
    o = port_lib.PortOracle(g.nv, g.off, g.adj, roots, nthreads=2)
    o.static()
    assert_levels(f.level64(), o.level())
    assert_sigma(f.sigma(), o.sigma(), o.level())
    assert_bc(f.bc(), o.bc())
    o.close()
    f.close()
    dg.close()


@pytest.mark.parametrize("reserve", [False, True])
def test_edge_that_comes_and_goes_on_the_device(sbc_lib, port_lib, reserve):
    g, roots, dg, f, hub, _, fresh, device = _start(200, 3)
    if reserve:
        dg.reserve(fresh[:1])
    for _ in range(20):
        device(fresh[:1])
        assert f.delete(fresh[:1])["inserted"] == 1
    for e in fresh[:40]:
        assert f.insert([e])["inserted"] == 1
    _check(port_lib, G.insert_edges(g, fresh[:40]), roots, dg, f)


def test_device_batch_in_the_room_that_deletions_left(sbc_lib, port_lib):
    g, roots, dg, f, hub, near, fresh, device = _start(200, 4)
    gone = np.array([(hub, x) for x in sorted(near)[:5]], dtype=np.int64)
    assert f.delete(gone)["inserted"] == 5
    device(fresh[:5])
    for e in fresh[5:40]:
        assert f.insert([e])["inserted"] == 1
    _check(port_lib, G.insert_edges(G.delete_edges(g, gone), fresh[:40]), roots, dg, f)


def test_device_batch_that_nobody_reserved_for(sbc_lib, port_lib):
    g, roots, dg, f, hub, _, fresh, device = _start(200, 6)
    device(fresh[:4])
    for e in fresh[4:40]:
        assert f.insert([e])["inserted"] == 1
    _check(port_lib, G.insert_edges(g, fresh[:40]), roots, dg, f)


def test_reserved_device_window_re_packs_once(sbc_lib, port_lib):
    g, roots, dg, f, hub, _, fresh, device = _start(200, 5)
    ins = fresh[:12].reshape(3, 4, 2)
    dg.reserve(ins[0])
    device(ins[0])
    for step in range(30):
        dg.reserve(ins[(step + 1) % 3])
        device(ins[(step + 1) % 3])
        assert f.delete(ins[step % 3])["inserted"] == 4
    assert dg.repacks() <= 1
    _check(port_lib, G.insert_edges(g, ins[30 % 3]), roots, dg, f)

"""The launch shape of a forest created without one: a CTA is no narrower than
its roots need, and a sparse graph's workers do not multiply the scratch."""
import ctypes as C

import numpy as np
import pytest

from streamingbc_gb300 import graphs as G
from streamingbc_gb300 import native

pytestmark = pytest.mark.gpu


def _threads(lib, forest):
    n = C.c_int(0)
    assert lib.sbc_update_variant_info(forest.variant, C.byref(n), None, None) == 0
    return n.value


@pytest.mark.parametrize("nv,ne,k,least", [(200, 800, 1, 512), (200, 800, 100, 512), (1024, 8192, 12, 512),
                                           (5000, 25000, 100, 512), (5000, 25000, 2000, 128),
                                           (70000, 600000, 5, 1024), (70000, 600000, 400, 1024)])
def test_width_follows_roots_and_slots(sbc_lib, nv, ne, k, least):
    g = G.er(nv, ne, seed=1)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    f = native.DeviceForest(dg, np.arange(k))
    assert _threads(sbc_lib, f) >= least
    f.close()
    dg.close()


@pytest.mark.parametrize("nv,ne,k", [(60000, 10000, 1216), (130000, 5000, 500), (3000, 6000, 2000)])
def test_scratch_of_sparse_graphs(sbc_lib, nv, ne, k):
    g = G.er(nv, ne, seed=2)
    dg = native.DeviceGraph(g.nv, g.off, g.adj)
    own = native.DeviceForest(dg, np.arange(k))
    wide = native.DeviceForest(dg, np.arange(k), variant=7)  # a worker per SM
    # twice that, or a quarter of a gigabyte
    extra = own.info()["bytes"] - wide.info()["bytes"]
    per = wide.info()["workers"] * 38 * nv
    assert extra <= max(1.02 * per, 2 ** 28)
    for f in (own, wide):
        f.close()
    dg.close()

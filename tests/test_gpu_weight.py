"""Child weights against division: within one unit in the last place over the
values that path counts and dependencies take, and the same result for those
they take when sums have wrapped or are not finite."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from streamingbc_gb300 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def weights(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("weight") / "child_weight.so")
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I" + build.CSRC, "-shared", "-o", so,
                        os.path.join(HERE, "c", "child_weight.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(so)

    def run(a, s):
        a, s = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(s, np.int64)
        w, q = np.empty_like(a), np.empty_like(a)
        p = [x.ctypes.data_as(C.c_void_p) for x in (a, s, w, q)]
        assert lib.child_weights(C.c_int(a.size), *p) == 0
        return w, q

    return run


def _ulps(w, q):
    return np.abs(w - q) / np.spacing(np.abs(q))


EDGES = np.array([1, 2, 3, 5, 7, 2**23 - 1, 2**23, 2**24 - 1, 2**24, 2**24 + 1, 2**31 - 1, 2**31, 2**52, 2**53 - 1, 2**53,
                  2**53 + 1, 2**53 + 3, 2**62, 2**63 - 1025, 2**63 - 513, 2**63 - 1], dtype=np.int64)


def test_over_the_range(weights):
    rng = np.random.default_rng(1)
    n = 1 << 21
    s = (2.0 ** rng.uniform(0, 63, n)).clip(max=2.0 ** 63 - 1024).astype(np.int64)
    a = 1.0 + np.where(rng.random(n) < 0.3, 0.0, 2.0 ** rng.uniform(-40, 60, n))
    a[: n // 8] = rng.integers(1, 1 << 20, n // 8)
    w, q = weights(a, s)
    assert np.array_equal(q, a / s.astype(np.float64))
    assert _ulps(w, q).max() <= 1.0
    # a difference of weights starts from ones that are equal to the last bit almost everywhere
    assert np.count_nonzero(w != q) <= n * 2.0 ** -30


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_edges_of_sigma(weights, sign):
    a = sign * np.array([1.0, 1.5, 3.0, 1 + 2.0 ** -52, 2.0 ** 53 - 1, 1e-3, 1e-300, 1e15, 1e300, 2.0 ** 1021, 1.7e308])
    aa, ss = (x.ravel() for x in np.meshgrid(a, EDGES))
    w, q = weights(aa, ss)
    assert np.array_equal(q, aa / ss.astype(np.float64))
    assert _ulps(w, q).max() <= 1.0


def test_wrapped_and_not_finite(weights):
    a = np.array([1.0, -1.0, 0.5, 1e300, -1e300, np.inf, -np.inf, np.nan, 0.0])
    s = np.array([0, -1, -5, -2**40, -2**63, 1, 3, 2**53 + 1, 2**63 - 1], dtype=np.int64)
    aa, ss = (x.ravel() for x in np.meshgrid(a, s))
    w, q = weights(aa, ss)
    same = (w == q) | (np.isnan(w) & np.isnan(q))
    assert same.all(), (aa[~same], ss[~same], w[~same], q[~same])

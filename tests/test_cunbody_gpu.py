"""The CUNBODY-compatible slot (bin/cunbody.h:11-33) exported by libsimgb:
ai = sum_j mj (xj - xi) / (|xj - xi|^2 + eps2)^{3/2}, driven as the reference's
_cunbody wrapper does (bin/cunbody.cpp:43-90: xj = xi = pos2, mj = 1, eps2 = 1e-23)."""
import ctypes

import numpy as np
import pytest

from simbuca_gb300 import abi

pytestmark = pytest.mark.gpu


def reference_sum(xj, mj, xi, eps2):
    d = xj[None, :, :] - xi[:, None, :]
    r2 = (d * d).sum(-1) + eps2
    w = np.where(r2 > 0, mj[None, :] / np.where(r2 > 0, r2, 1.0) ** 1.5, 0.0)
    return (d * w[:, :, None]).sum(1)


def call(fn, xj, mj, xi, eps2):
    L = abi.load()
    ai = np.zeros((len(xi), 3))
    getattr(L, fn)(abi.dptr(xj), abi.dptr(mj), abi.dptr(xi), eps2, abi.dptr(ai), len(xi), len(xj))
    return ai


def test_wrapper_usage():
    rng = np.random.default_rng(1)
    n = 700
    x = rng.normal(0, 5e-4, (n, 3))
    m = np.ones(n)
    eps2 = float(np.float32(1e-23))  # the wrapper keeps eps in a float (bin/cunbody.h:49)
    ai = call("cunbody1_force", x, m, x.copy(), eps2)
    ref = reference_sum(x, m, x, eps2)
    np.testing.assert_allclose(ai, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


def test_begin_end_distinct_sets():
    rng = np.random.default_rng(2)
    xj = rng.normal(0, 1e-3, (300, 3))
    mj = rng.uniform(0.5, 2.0, 300)
    xi = rng.normal(0, 1e-3, (129, 3))
    L = abi.load()
    ai = np.zeros((129, 3))
    args = (abi.dptr(xj), abi.dptr(mj), abi.dptr(xi), 1e-12, abi.dptr(ai), 129, 300)
    L.cunbody1_force_begin(*args)
    L.cunbody1_force_end(*args)
    ref = reference_sum(xj, mj, xi, 1e-12)
    np.testing.assert_allclose(ai, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


@pytest.mark.parametrize("ni,nj", [(1, 1), (33, 33), (128, 128), (129, 129), (1000, 1000),
                                   (1, 700), (129, 3000), (5, 128)])
@pytest.mark.parametrize("eps2", [0.0, 1e-12])
def test_set_sizes_and_coincident_pairs(ni, nj, eps2):
    """One array as both sets takes each unordered pair once, different sets take j-chunks:
    tile edges of both, with two ions at one place (no contribution without softening) and
    with equal and unequal masses.  The slot's tolerance, as above."""
    rng = np.random.default_rng(ni + nj)
    xj = rng.normal(0, 1e-3, (nj, 3))
    if nj > 2:
        xj[nj // 2] = xj[0]
    same = ni == nj
    xi = xj.copy() if same else rng.normal(0, 1e-3, (ni, 3))
    if not same:
        xi[0] = xj[1]
    for mj in (np.full(nj, 1.5), rng.uniform(0.5, 2.0, nj)):
        ai = call("cunbody1_force", xj, mj, xi, eps2)
        ref = reference_sum(xj, mj, xi, eps2)
        np.testing.assert_allclose(ai, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


def test_scratch_of_a_large_set_is_given_back():
    """Partial sums of one set against itself: 0.8 GB at 65,536 ions while the call runs, at most
    256 MB of them kept for the next one (with the buffers and the runtime's own granularity:
    512 MB); sums checked on a few rows."""
    torch = pytest.importorskip("torch")
    n = 65536
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1e-3, (n, 3))
    mj = np.ones(n)
    call("cunbody1_force", x[:256].copy(), mj[:256], x[:256].copy(), 0.0)  # the context exists
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ai = call("cunbody1_force", x, mj, x.copy(), 0.0)
    assert before - torch.cuda.mem_get_info()[0] <= 512 << 20
    for i in (0, 127, 128, 40000, n - 1):
        d = np.delete(x, i, axis=0) - x[i]
        ref = (d / (d * d).sum(1)[:, None] ** 1.5).sum(0)
        np.testing.assert_allclose(ai[i], ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


@pytest.mark.parametrize("ni,nj", [(1, 1), (2, 2), (31, 31), (32, 32), (33, 33), (1, 128), (300, 128),
                                   (300, 129), (7, 1), (1, 0), (64, 33)])
def test_one_launch_and_two_launch_sizes(ni, nj):
    """Up to 128 j-ions the sums go straight to ai, beyond through partial sums; one set against
    itself takes unordered pairs above 32 ions.  Both sides of each line; no j-ions give 0."""
    rng = np.random.default_rng(100 * ni + nj)
    xj = rng.normal(0, 1e-3, (nj, 3))
    xi = xj.copy() if ni == nj else rng.normal(0, 1e-3, (ni, 3))
    mj = rng.uniform(0.5, 2.0, nj)
    for _ in range(2):
        ai = call("cunbody1_force", xj, mj, xi, 1e-14)
        ref = reference_sum(xj, mj, xi, 1e-14)
        np.testing.assert_allclose(ai, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


def test_a_single_ion_takes_one_launch():
    """The call time of one ion against itself, which two launches made 10 us longer, against
    that of 33 ions, which take two: shorter by at least a launch's few microseconds."""
    import time

    def best(n):
        x, m = np.random.default_rng(n).normal(0, 1e-3, (n, 3)), np.ones(n)
        t = []
        for _ in range(200):
            t0 = time.perf_counter()
            call("cunbody1_force", x, m, x, 1e-14)
            t.append(time.perf_counter() - t0)
        return min(t) * 1e6

    one, two = best(1), best(33)
    print(one, two)
    assert one <= two - 2.0

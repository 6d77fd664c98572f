"""The FP64 sums over unordered pairs at the sizes where their items change: tile pairs in
four, two or one parts (smallest sets), 128 x 32 items (above ~4,400 ions), and the edges of
the 32-ion tiles; equal and mixed charges, against the oracle."""
import numpy as np
import pytest

import oracle
from simbuca_gb300 import configs
from simbuca_gb300.abi import SG_PREC_FP64
from simbuca_gb300.api import Batch
from helpers import kq_of, rel_err_per_ion, summary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [2, 33, 64, 200, 257, 300, 417, 600, 700, 1000, 4416, 4500])
def test_sums_against_the_oracle(ctx, n, mixed):
    """1e-12 of the ion's sum, as for every size: FP64 terms to an ulp or so, sums of n terms
    whose rounding grows with sqrt(n) at most (sqrt(4,500) 1.1e-16 = 7e-15, times the
    cancellation of an ion's terms, up to ~100 near the centre)."""
    rng = np.random.default_rng(n)
    pos = rng.normal(0, 5e-4, (n, 3))
    q = rng.choice([1.0, 2.0, 3.0], n) if mixed else np.ones(n)
    kq = kq_of(np.full(n, 132.905 * oracle.AMU), q)
    a = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP64)
    first, last = min(n, 64), max(0, n - 64)
    for lo, hi in ((0, first), (last, n)):
        ref = oracle.coulomb_kq_rows(pos, q, kq, lo, hi)
        e = rel_err_per_ion(a[lo:hi], ref)
        assert e.max() <= 1e-12, (n, summary(e))


def device_bytes_taken(make):
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    b = make()
    return b, before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("counts", [[131072] * 64, [131072] + [8192] * 512])
def test_memory_of_large_batches(ctx, counts):
    """A slot per i-block of the largest cloud for every ion of the batch would be 200 to 275 GB
    here: such batches sum ordered pairs.  State, stages and coordinates are ~0.9 kB an ion,
    the ordered pairs' slots at most 32 x 24 B: 2 kB an ion, and what a context sets aside."""
    small = lambda: Batch(ctx, [64], [configs.penning_field()],
                          [configs.ode(1e-9, 1e-15, 1e-9, 1e-6)], SG_PREC_FP64)
    small()
    b, taken = device_bytes_taken(lambda: Batch(
        ctx, counts, [configs.penning_field()] * len(counts),
        [configs.ode(1e-9, 1e-15, 1e-9, 1e-6)] * len(counts), SG_PREC_FP64))
    print(len(counts), "clouds", taken / 1e9, "GB")
    assert taken <= 2048 * sum(counts) + (1 << 30)
    small()  # gives the memory back


@pytest.mark.parametrize("n", [131072, 131073])
def test_both_sides_of_the_largest_unordered_cloud(ctx, n):
    """131,072 ions are the most that take unordered pairs, one more takes ordered ones; rows at
    the first, an inner and the last block edge against the oracle, bound as above."""
    rng = np.random.default_rng(n)
    pos = rng.normal(0, 1e-3, (n, 3))
    q = rng.choice([1.0, 2.0], n)
    kq = kq_of(np.full(n, 132.905 * oracle.AMU), q)
    a = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP64)
    for lo in (0, 65536 - 8, n - 16):
        e = rel_err_per_ion(a[lo:lo + 16], oracle.coulomb_kq_rows(pos, q, kq, lo, lo + 16))
        assert e.max() <= 1e-12, (n, lo, summary(e))


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [6001, 8193, 12345, 20001])
def test_items_of_several_tiles_against_the_oracle(ctx, n, mixed):
    """Above ~6,300 ions an item is several j-tiles (K = 3 at 8,193 ions, 20 at 20,001), the last
    one ragged: every ion of the first, a middle and the last i-block, bound as above."""
    rng = np.random.default_rng(n)
    pos = rng.normal(0, 5e-4, (n, 3))
    q = rng.choice([1.0, 2.0, 3.0], n) if mixed else np.ones(n)
    kq = kq_of(np.full(n, 132.905 * oracle.AMU), q)
    a = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP64)
    mid = n // 2 // 128 * 128
    for lo, hi in ((0, 160), (mid - 32, mid + 160), (n - 160, n)):
        e = rel_err_per_ion(a[lo:hi], oracle.coulomb_kq_rows(pos, q, kq, lo, hi))
        assert e.max() <= 1e-12, (n, lo, summary(e))

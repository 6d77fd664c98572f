"""The FP64 sums over unordered pairs at the sizes where their items change: tile pairs in
four, two or one parts (smallest sets), 128 x 32 items (above ~4,400 ions), and the edges of
the 32-ion tiles; equal and mixed charges, against the oracle."""
import numpy as np
import pytest

import oracle
from simbuca_gb300.abi import SG_PREC_FP64
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

"""Contexts in threads of one program: each has its own stream and buffers, and integrates as
it does alone, whatever forms run beside each other on the device -- the wide form of small
clouds (a cooperative launch, whose CTAs wait for each other with a limit), clusters, leaf
pairs, FP64 tiles, and the CUNBODY slot of the process."""
import threading

import numpy as np
import pytest

from simbuca_gb300 import abi, configs
from simbuca_gb300.abi import SG_PREC_FP32C, SG_PREC_FP64
from simbuca_gb300.api import Batch, Context

pytestmark = pytest.mark.gpu


def integrate(counts, prec, attempts, rounds):
    """Fixed steps in a context of its own; the last state and the form the batch took."""
    ctx = Context(0)
    rng = configs.rng_for(sum(counts))
    clouds = [configs.gaussian_cloud(rng, n, 5e-4, 300.0, np.full(n, configs.M_CS)) for n in counts]
    fp = configs.penning_field(quad=(0.5, configs.nu_c(configs.M_CS), 0.0, 0.0, 1.0), delta=1e3)
    b = Batch(ctx, counts, [fp] * len(counts), [configs.ode(1e-9, 1e-15, 1e-9, 1.0, adaptive=False)] * len(counts), prec)
    args = [np.concatenate([getattr(c, k) for c in clouds]) for k in ("pos", "vel", "mass")]
    for _ in range(rounds):
        b.upload(*args, np.concatenate([c.charge for c in clouds]).astype(np.int32))
        for _ in range(attempts // 5):
            b.attempts(5)
        info = b.info()
        assert all(i["status"] == abi.SG_OK and i["steps"] == attempts for i in info)
    out = b.download(), b.fused()
    ctx.close()
    return out


WIDE = ([1000], SG_PREC_FP32C, 40, 10)
WIDE_SHARED = ([4000], SG_PREC_FP32C, 20, 10)
CLUSTER = ([300], SG_PREC_FP32C, 40, 10)
LEAVES = ([30000], SG_PREC_FP32C, 10, 6)
PAIRS64 = ([9000], SG_PREC_FP64, 5, 6)


@pytest.mark.parametrize("jobs", [(WIDE, WIDE), (WIDE, WIDE_SHARED, CLUSTER), (WIDE, LEAVES), (WIDE_SHARED, PAIRS64, LEAVES)],
                         ids=["two_wide", "wide_and_cluster", "wide_and_leaves", "wide_fp64_leaves"])
def test_each_context_integrates_as_it_does_alone(jobs):
    alone = [integrate(*j) for j in jobs]
    assert alone[0][1] > 16
    got, errors = [None] * len(jobs), []

    def work(k):
        try:
            got[k] = integrate(*jobs[k])
        except Exception as e:  # reported by the test
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (state, form), (ref, ref_form) in zip(got, alone):
        assert form == ref_form
        assert np.array_equal(state[0], ref[0]) and np.array_equal(state[1], ref[1])

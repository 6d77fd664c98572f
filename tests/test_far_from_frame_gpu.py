"""Close pairs of a cloud that has left the frame it was uploaded in (a TOF kick, a drift):
the FP32c frame coordinates are then large numbers, and a close pair's distance is a small
difference of two of them."""
import numpy as np
import pytest

import oracle
from simbuca_gb300 import abi, configs
from simbuca_gb300.abi import SG_PREC_FP32C, SG_PREC_FP64
from simbuca_gb300.api import Batch
from helpers import kq_of

pytestmark = pytest.mark.gpu

N, L = 400, 1e-3
SEP = np.array([1.2e-5, 3e-5, 1e-4, 1e-3])  # of the spread


@pytest.fixture(params=["fused", "plain", "sorted", "leaf"])
def form(request, ctx):
    ctx.set_fused(request.param == "fused")
    ctx.set_coulomb_variant({"fused": -1, "plain": 11, "sorted": 9, "leaf": 17}[request.param])
    yield request.param
    ctx.set_fused(True)
    ctx.set_coulomb_variant(-1)


@pytest.mark.parametrize("drift", [30.0, 1e4])
def test_close_pairs_after_a_drift(ctx, form, drift):
    """One step with a common velocity along x that carries the cloud `drift` spreads away from
    its frame, pairs separated along (0, 1, 0) turned by 45 degrees into x: the error of the x
    difference enters the y force at first order, and y velocities start at 0, so the step's
    y velocity is the force (the step's own displacement of a pair is below 1e-9 of its
    distance).  Both forms see the same SI coordinates (rounded alike at the drifted place).
    A pair taken in float-float is at least 1e-5 |u| apart and its coordinates are good to
    2^-49 |u| each, its distance to 4e-10 and its force to 1e-9 (the other ions' FP32 terms are
    4e-4 of it and add 1e-10): 2e-9 for the pairs' ions, the FP32c bound of 1e-6 for all."""
    rng = np.random.default_rng(11)
    pos = rng.normal(0, L, (N, 3))
    for k, s in enumerate(np.repeat(SEP, 4)):
        pos[2 * k + 1] = pos[2 * k] + s * L * np.array([1.0, 1.0, 0.0]) / np.sqrt(2)
    h = 1e-9
    vel = np.zeros((N, 3))
    vel[:, 0] = drift * L / h
    fp = abi.FieldParams()
    fp.flags = abi.SG_F_COULOMB
    # a pair 1.2e-8 m apart accelerates by k_e e^2 / (m r^2) = 7e12 m/s^2 without the scale: h^2
    # times that is 7e-6 m, with it 7e-18 m, below 1e-9 of 1.2e-8 m
    fp.coulomb_scale = 1e-12
    mass = np.full(N, configs.M_CS * oracle.AMU)
    full = ctx.coulomb_accel(pos, np.ones(N), fp.coulomb_scale * kq_of(mass, np.ones(N)), SG_PREC_FP64)
    out = []
    for prec in (SG_PREC_FP32C, SG_PREC_FP64):
        b = Batch(ctx, [N], [fp], [configs.ode(1e-9, 1e-15, h, 1.0, adaptive=False)], prec)
        if prec == SG_PREC_FP32C:
            assert (b.fused() > 0) == (form == "fused")
        b.upload(pos, vel, mass, np.ones(N, np.int32))
        b.attempts(1)
        out.append(b.download()[1])
    a, r = out[0][:, 1:], out[1][:, 1:]
    e = np.linalg.norm(a - r, axis=1) / (h * np.linalg.norm(full, axis=1))
    print(form, drift, "pairs", e[:8 * len(SEP)].max(), "all", e.max())
    assert e[:8 * len(SEP)].max() <= 2e-9
    assert e.max() <= 1e-6

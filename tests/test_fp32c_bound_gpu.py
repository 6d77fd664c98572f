"""The FP32-compensated form's per-ion bound (relative force error <= 1e-6 against the
FP64 direct sum of bin/force.cpp:147-174) beyond the two clouds its far fix-up threshold
was first calibrated on, and the in-run check that measures the error while a cloud
evolves.

Sampled rows (random ions, the ions nearest the centre -- where the net force is small
next to the far terms -- and both ions of the closest pairs) are compared with the
oracle's FP64 rows on a 262,144-ion uniform spheroid, a 1,048,576-ion Gaussian cloud,
the 65,536-ion Gaussian cloud at 1 K, and a 65,536-ion cloud 125 times denser than
that one."""
import os

import numpy as np
import pytest

import oracle
from simbuca_gb300 import configs
from simbuca_gb300.abi import SG_PREC_FP32C, SG_PREC_FP64
from simbuca_gb300.api import Batch
from helpers import kq_of, rel_err_per_ion, summary

pytestmark = pytest.mark.gpu
BOUND = 1e-6


@pytest.fixture(scope="module", autouse=True)
def _oracle():
    oracle.build()
    oracle.set_threads(os.cpu_count() or 4)


def sampled_rows(pos, n_random=40, n_central=16, n_close=16, seed=1):
    n = len(pos)
    rng = np.random.default_rng(seed)
    c = pos.mean(0)
    r2 = ((pos - c) ** 2).sum(1)
    # closest pairs: neighbours in a lexicographic order of a fine grid
    order = np.lexsort(np.floor((pos - pos.min(0)) / 2e-6).T)
    d = np.linalg.norm(np.diff(pos[order], axis=0), axis=1)
    close = np.argsort(d)[:n_close]
    rows = np.concatenate([rng.choice(n, n_random, replace=False), np.argsort(r2)[:n_central],
                           order[close], order[close + 1]])
    return np.unique(rows)


def check_rows(ctx, pos, q, mass, label):
    kq = kq_of(mass, q)
    a = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP32C)
    assert np.isfinite(a).all()
    rows = sampled_rows(pos)
    ref = np.stack([oracle.coulomb_kq_rows(pos, q, kq, int(i), int(i) + 1)[0] for i in rows])
    e = rel_err_per_ion(a[rows], ref)
    print(label, summary(e))
    assert e.max() <= BOUND, (label, summary(e))


def test_spheroid_262k(ctx):
    c = configs.spheroid_cloud(configs.rng_for(12), 1 << 18, 2e-3, 4e-3, 1.0, configs.M_CS)
    check_rows(ctx, c.pos, c.charge.astype(np.float64), c.mass, "spheroid 262k")


def test_gaussian_1m(ctx):
    n = 1 << 20
    c = configs.gaussian_cloud(configs.rng_for(13), n, 1e-3, 300.0, np.full(n, configs.M_CS))
    check_rows(ctx, c.pos, c.charge.astype(np.float64), c.mass, "gaussian 1M")


def test_gaussian_65k_cold(ctx):
    n = 65536
    c = configs.gaussian_cloud(configs.rng_for(14), n, 1e-3, 1.0, np.full(n, configs.M_CS))
    check_rows(ctx, c.pos, c.charge.astype(np.float64), c.mass, "65k at 1 K")


def test_gaussian_65k_dense(ctx):
    n = 65536
    c = configs.gaussian_cloud(configs.rng_for(15), n, 0.2e-3, 1.0, np.full(n, configs.M_CS))
    check_rows(ctx, c.pos, c.charge.astype(np.float64), c.mass, "65k, sigma 0.2 mm")


def test_in_run_check_on_the_65k_workload(ctx):
    """The check runs inside the attempt loop at its default interval: on the 65,536-ion
    workload it finds no probe above the bound and keeps the density prior."""
    w = configs.penning_65k()
    c = w.clouds[0]
    b = Batch(ctx, [len(c.mass)], w.fields, w.odes, SG_PREC_FP32C)
    b.set_force_check(2)
    b.upload(c.pos, c.vel, c.mass, c.charge)
    for _ in range(12):
        b.step()
    rec = b.force_check()[0]
    print(rec)
    assert rec["checks"] >= 6 and rec["probes"] == 8 * rec["checks"]
    assert rec["breaches"] == 0 and 0.0 < rec["max_err"] <= BOUND
    assert rec["kfar"] <= rec["kfar_prior"]


def test_in_run_check_repairs_a_far_threshold_set_too_high(ctx):
    """With the far fix-up switched off (prior kfar = 1e6) the central ions of the
    1,048,576-ion spheroid carry the hi-only far error (~1.1e-6 before the fix-up
    existed).  The first check measures c on them and lowers kfar to 5e-7 / c; the
    attempts after it are checked within the bound."""
    w = configs.spheroid_1m()
    c = w.clouds[0]
    b = Batch(ctx, [len(c.mass)], w.fields, w.odes, SG_PREC_FP32C)
    b.set_far_threshold(1e6)
    b.set_force_check(1)
    b.upload(c.pos, c.vel, c.mass, c.charge)
    b.attempts(1)
    first = b.force_check()[0]
    print("first", first)
    assert first["checks"] == 1 and first["kfar_prior"] == pytest.approx(1e6)
    assert first["c_far"] > 2e-7                      # the hi-only far error is measured
    assert first["kfar"] == pytest.approx(max(5e-7 / first["c_far"], 0.05), rel=1e-5)
    b.attempts(2)
    rec = b.force_check()[0]
    print("after", rec)
    assert rec["checks"] == 3
    assert rec["last_err"] <= BOUND and rec["kfar"] <= first["kfar"] * (1 + 1e-6)


def planted(n, seed):
    """A Gaussian cloud (sigma 1 mm) whose ion 0 sits at the centre between three pairs of
    ions at about 0.9 of the mean ion spacing on each axis, the other ions moved out of a
    5-spacing ball around it: six strong pair terms that nearly cancel, outside the
    close-pair radius (0.6 spacings), with a net force of 2 % of one of those terms: ion 0
    is summed in FP32 and flagged by the conditioning test."""
    c = configs.gaussian_cloud(configs.rng_for(seed), n, 1e-3, 300.0, np.full(n, configs.M_CS))
    pos = c.pos.copy()
    ctr = pos.mean(0)
    spacing = np.cbrt((2 * np.pi) ** 1.5 * np.prod(pos.std(0)) / n)
    r = pos - ctr
    d = np.linalg.norm(r, axis=1)
    inner = d < 5 * spacing
    pos[inner] = ctr + r[inner] * ((5 * spacing + d[inner]) / d[inner])[:, None]
    # the spacing the library's frame takes (from the moved cloud's spreads)
    spacing = np.cbrt((2 * np.pi) ** 1.5 * np.prod(pos.std(0)) / n)
    # ion 0 at the centre; on each axis one neighbour at -a and one at +a_ax, a_ax chosen
    # so that the pair cancels the rest of the cloud's field there up to a net force of
    # 2 % of one neighbour's term
    q = c.charge.astype(np.float64)
    a = 0.9 * spacing
    pos[0] = ctr
    d = ctr - pos[7:]
    bg = (q[7:, None] * d / ((d * d).sum(1) ** 1.5)[:, None]).sum(0)
    target = 0.02 / a ** 2 * np.ones(3) / np.sqrt(3.0)
    for ax in range(3):
        # field on ion 0 along ax: q/a^2 - q/a_ax^2 + bg_ax = target_ax
        inv2 = 1.0 / a ** 2 + (bg[ax] - target[ax]) / q[1 + 2 * ax]
        pos[1 + 2 * ax] = ctr
        pos[1 + 2 * ax, ax] += 1.0 / np.sqrt(inv2)
        pos[2 + 2 * ax] = ctr
        pos[2 + 2 * ax, ax] -= a
    return pos, q, c.mass


@pytest.mark.parametrize("n,variant", [(300, -1), (4096, -1), (20000, -1), (20000, 9),
                                       (65536, 14)])
def test_flagged_ion_gets_its_exact_row(ctx, n, variant):
    """An ion whose FP32 terms cancel keeps, after its dominant pairs alone are re-taken in
    FP64, the rounding of the FP32 additions made while they were in its partial sums
    (~1e-7 of its strongest term: up to ~5e-6 of its net force in the 512-cloud scan).
    A flagged ion's sum is therefore replaced by its FP64 row: in-block for batches of up
    to 8,192 ions, spread over 16 work units beyond; for the plain and k-d ordered shapes."""
    pos, q, mass = planted(n, 20 + n % 7)
    kq = kq_of(mass, q)
    assert np.isfinite(pos).all()
    try:
        ctx.set_coulomb_variant(variant)
        a32 = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP32C)
    finally:
        ctx.set_coulomb_variant(-1)
    a64 = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP64)
    ref = oracle.coulomb_kq_rows(pos, q, kq, 0, 1)[0]
    e = rel_err_per_ion(a32, a64)
    e0 = float(np.linalg.norm(a32[0] - ref) / np.linalg.norm(ref))
    print(n, variant, "planted ion", e0, "all ions", summary(e))
    assert e0 <= 1e-12
    assert e.max() <= BOUND


@pytest.mark.parametrize("n", [9000, 70000])
def test_more_flagged_ions_than_the_unit_list_holds(ctx, n):
    """A lattice of alternating charges: the terms of an inner ion cancel, so that most ions
    are flagged -- more work units than their list holds, the rest whole.  Every flagged
    row is exact to FP64 rounding: n terms whose magnitudes add up to ~4 pi R in units of a
    neighbour's field (R = 21, 41 spacings across): 1e-16 sqrt(n) 250 < 1e-11 of that field,
    in either form's order of summation.  The others keep the FP32c bound (of fields of the
    order of a neighbour's)."""
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = 1e-5 * g.astype(np.float64)
    q = np.where(g.sum(1) % 2 == 0, 1.0, -1.0)
    kq = np.abs(kq_of(np.full(n, configs.M_CS), np.ones(n)))
    ctx.fixup_count()
    a32 = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP32C)
    flagged = ctx.fixup_count()
    a64 = ctx.coulomb_accel(pos, q, kq, SG_PREC_FP64)
    err = np.abs(a32 - a64).max(1) / (kq[0] / 1e-10)
    print(n, "flagged", flagged, "largest", err.max())
    assert flagged > 4000
    assert err.max() <= BOUND
    assert (err <= 1e-11).sum() >= flagged

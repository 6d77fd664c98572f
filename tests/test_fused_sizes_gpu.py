"""The fused small-cloud kernel at the sizes where its layout changes: clouds of fewer ions
than CTAs take, the CTA's rows whole 16-byte words or not, one and two slots per thread
(1,344 ions on 16 CTAs), each with an ion at the centre whose terms cancel (its row comes
from the FP64 loop) and a close pair."""
import numpy as np
import pytest

from simbuca_gb300 import configs
from simbuca_gb300.abi import SG_PREC_FP32C, SG_PREC_FP64
from simbuca_gb300.api import Batch

pytestmark = pytest.mark.gpu


def fixed_steps(ctx, pos, vel, mass, charge, prec, fused, steps):
    fp = configs.penning_field(quad=(0.5, configs.nu_c(132.905), 0.0, 0.0, 1.0), delta=1e3)
    ctx.set_fused(fused)
    try:
        b = Batch(ctx, [len(mass)], [fp], [configs.ode(1e-9, 1e-15, 2e-9, 1.0, adaptive=False)], prec)
        b.upload(pos, vel, mass, charge)
        assert (b.fused() > 0) == (fused == 2 and prec == SG_PREC_FP32C)
        b.run(max_attempts=steps)
        return b.download()
    finally:
        ctx.set_fused(1)


@pytest.mark.parametrize("n", [3, 4, 5, 16, 17, 64, 65, 300, 1344, 1345])
@pytest.mark.parametrize("charges", ["one", "mixed"])
def test_sizes_against_fp64(ctx, n, charges):
    """Eight fixed steps against the FP64 form.  The FP32c force is within 1e-6 of the ion's
    own Coulomb force; over 16 ns the Coulomb force moves an ion by less than 1e-3 of the
    cloud's extent, so positions agree to 1e-9 of it and velocities (Coulomb part below
    the thermal speed by the same reasoning) to 1e-8 of theirs."""
    c = configs.gaussian_cloud(configs.rng_for(70 + n), n, 0.5e-3, 300.0,
                               np.full(n, configs.M_CS))
    pos, q = c.pos.copy(), c.charge.copy()
    pos[0] = pos.mean(0)                      # cancelling terms
    if n >= 16:
        pos[2] = pos[1] + [4e-7, 0.0, 2e-7]   # a close pair
    if charges == "mixed":
        q[::3] = 2
    out = [fixed_steps(ctx, pos, c.vel, c.mass, q, prec, 2, 8) for prec in (SG_PREC_FP32C, SG_PREC_FP64)]
    ep = np.abs(out[0][0] - out[1][0]).max() / np.abs(out[1][0]).max()
    ev = np.abs(out[0][1] - out[1][1]).max() / np.abs(out[1][1]).max()
    print(n, charges, ep, ev)
    assert ep <= 1e-9 and ev <= 1e-8

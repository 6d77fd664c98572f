"""Performance cases: the work a simulation has this package do, through its public
entry points (`Context`, `Batch`, and the C entry points for device pointers and for the
CUNBODY slot).

A case is a dict with its `kind`:

  integrate  resident clouds advanced `attempts` integrator attempts (or one accepted
             step when attempts is 0, the `step()` call of a host-driven loop), then
             read back.  Adaptive runs start at a picosecond step, as a user without a
             guess does, and let the controller grow it; the others use the fixed-step
             mode (trajectory comparisons).
  coupled    a host program that edits the state between steps: set_state, a step,
             download, every pass.
  force      one force() call from host arrays (field terms and Coulomb sum), FP64.
  device     the Coulomb sum on the caller's device buffers, no allocation, FP64.
  cunbody    the reference's CUNBODY library slot: host arrays, softened sum, FP64.
  train      training of the step-size proposer network on logged step histories.

Inputs are seeded synthetic ion clouds in the traps of the benchmark workloads.
"""
import math

import numpy as np
import torch

from simbuca_gb300 import abi
from simbuca_gb300.api import Batch, Context

AMU, E, KB = 1.6605402e-27, 1.60217733e-19, 1.3806504e-23
KE, PI = 8.987551787e9, 3.14159265358979323
MASS = 132.905
FP64, FP32C = 0, 1


def listed():
    return [
        # a few hundred ions stepped one accepted step at a time by the host: latency only
        {"name": "step_300", "kind": "integrate", "trap": "penning", "n": 300, "clouds": 1,
         "precision": FP32C, "method": 5, "adaptive": True, "h": 1e-12, "attempts": 0,
         "sigma": 5e-4, "temp": 300.0, "seed0": 0},
        # the small cloud of the benchmark between two outputs
        {"name": "run_1k", "kind": "integrate", "trap": "penning", "n": 1000, "clouds": 1,
         "precision": FP32C, "method": 5, "adaptive": False, "h": 4e-9, "attempts": 8,
         "sigma": 5e-4, "temp": 300.0, "seed0": 0},
        # the same cloud in the plain FP64 form under the step-size controller
        {"name": "run_1k_fp64", "kind": "integrate", "trap": "penning", "n": 1000, "clouds": 1,
         "precision": FP64, "method": 5, "adaptive": True, "h": 1e-11, "attempts": 2,
         "sigma": 5e-4, "temp": 300.0, "seed0": 0},
        # a host program that exchanges a 4,096-ion state with the device every step
        {"name": "coupled_4k", "kind": "coupled", "trap": "driven", "n": 4096, "clouds": 1,
         "precision": FP32C, "method": 5, "adaptive": False, "h": 2e-9, "attempts": 0,
         "sigma": 5e-4, "temp": 300.0, "seed0": 4},
        # the reference's own trap with mixed charges under its "RungaKutta4"; odd size
        {"name": "paul_20k_ck", "kind": "integrate", "trap": "paul", "n": 20001, "clouds": 1,
         "precision": FP32C, "method": 4, "adaptive": False, "h": 2e-9, "attempts": 1,
         "sigma": 1e-3, "temp": 300.0, "seed0": 5},
        # the headline workload: 65,536 driven, cooled ions of two masses, one step
        {"name": "penning_65k", "kind": "integrate", "trap": "driven", "n": 65536, "clouds": 1,
         "precision": FP32C, "method": 5, "adaptive": False, "h": 1e-9, "attempts": 1,
         "sigma": 1e-3, "temp": 300.0, "seed0": 1},
        # a large cold uniform spheroid, ragged size
        {"name": "spheroid_500k", "kind": "integrate", "trap": "spheroid", "n": 500009,
         "clouds": 1, "precision": FP32C, "method": 5, "adaptive": False, "h": 2.5e-10,
         "attempts": 1, "sigma": 2e-3, "temp": 1.0, "seed0": 2},
        # a frequency scan: uneven independent clouds (64 to 8,192 ions) in one batch
        {"name": "scan_128", "kind": "integrate", "trap": "driven", "n": 8192, "clouds": 128,
         "precision": FP32C, "method": 5, "adaptive": False, "h": 4e-9, "attempts": 4,
         "sigma": 5e-4, "temp": 300.0, "seed0": 3},
        # one force() call of a host integrator (default precision), odd size
        {"name": "force_5k_fp64", "kind": "force", "trap": "paul", "n": 5003, "clouds": 1,
         "precision": FP64, "sigma": 5e-4, "temp": 300.0, "seed0": 6},
        # a plug-in's Coulomb sum on device buffers: short enough that launches count
        {"name": "device_2k_fp64", "kind": "device", "n": 2048, "sigma": 5e-4, "seed0": 7},
        # the reference compiled for CUNBODY, linked against this library
        {"name": "cunbody_10k_fp64", "kind": "cunbody", "ni": 10007, "nj": 10007,
         "sigma": 5e-4, "seed0": 8},
        # proposer training, a stretch of minibatch iterations
        {"name": "train_256", "kind": "train", "n": 2000, "batch": 256, "iters": 8, "seed0": 9},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    k = rng.choice(["small", "small", "run", "run64", "coupled", "paul", "large", "large", "scan",
                    "force", "device", "cunbody", "train"])
    s = rng.randrange(1 << 20)
    base = {"kind": "integrate", "clouds": 1, "precision": FP32C, "method": 5, "sigma": 5e-4,
            "temp": 300.0, "seed0": s}
    if k == "small":
        return {**base, "trap": rng.choice(["penning", "driven"]), "n": _log(rng, 32, 2048),
                "adaptive": True, "h": 1e-12, "attempts": 0}
    if k == "run":
        return {**base, "trap": rng.choice(["penning", "driven"]), "n": _log(rng, 64, 12000),
                "adaptive": False, "h": 2e-9, "attempts": rng.randrange(2, 17)}
    if k == "run64":
        return {**base, "precision": FP64, "trap": rng.choice(["penning", "paul"]),
                "n": _log(rng, 32, 4000), "adaptive": True, "h": 1e-11,
                "attempts": rng.randrange(1, 3)}
    if k == "coupled":
        return {**base, "kind": "coupled", "trap": "driven", "n": _log(rng, 512, 40000),
                "adaptive": False, "h": 2e-9, "attempts": 0}
    if k == "paul":
        return {**base, "trap": "paul", "n": _log(rng, 2000, 60000), "sigma": 1e-3,
                "method": rng.choice([4, 1]), "adaptive": False, "h": 2e-9,
                "attempts": rng.randrange(1, 3)}
    if k == "large":
        trap = rng.choice(["driven", "spheroid"])
        n = _log(rng, 12000, 300000)
        if trap == "driven":
            return {**base, "trap": trap, "n": n, "sigma": 1e-3, "adaptive": False, "h": 1e-9,
                    "attempts": 1}
        return {**base, "trap": trap, "n": n, "sigma": 2e-3, "temp": 1.0, "adaptive": False,
                "h": 2.5e-10, "attempts": 1}
    if k == "scan":
        return {**base, "trap": "driven", "n": _log(rng, 300, 8192),
                "clouds": rng.randrange(8, 200), "adaptive": False, "h": 4e-9,
                "attempts": rng.randrange(1, 5)}
    if k == "force":
        return {"kind": "force", "trap": rng.choice(["paul", "penning"]), "clouds": 1,
                "n": _log(rng, 100, 12000), "precision": FP64, "sigma": 5e-4, "temp": 300.0,
                "seed0": s}
    if k == "device":
        return {"kind": "device", "n": _log(rng, 32, 8192), "sigma": 5e-4, "seed0": s}
    if k == "cunbody":
        return {"kind": "cunbody", "ni": _log(rng, 128, 16000), "nj": _log(rng, 128, 16000),
                "sigma": 5e-4, "seed0": s}
    return {"kind": "train", "n": rng.randrange(300, 4000), "batch": rng.choice([64, 128, 256]),
            "iters": rng.randrange(2, 11), "seed0": s}


# ---- inputs ------------------------------------------------------------------------
def _rng(case, seed):
    return np.random.Generator(np.random.Philox([case["seed0"], seed]))


def _counts(case):
    """Ions per cloud: one cloud of n, or log-uniform in [64, n] from the case itself."""
    if case["clouds"] == 1:
        return [case["n"]]
    r = np.random.Generator(np.random.Philox(case["seed0"]))
    lo, hi = math.log(min(64, case["n"])), math.log(case["n"])
    return [int(v) for v in np.floor(np.exp(r.uniform(lo, hi, case["clouds"]))).clip(1)]


def _cloud(case, seed):
    rng = _rng(case, seed)
    n = sum(_counts(case))
    if case["trap"] == "spheroid":
        out = []
        while sum(map(len, out)) < n:
            u = rng.uniform(-1.0, 1.0, (2 * n + 16, 3))
            out.append(u[(u * u).sum(1) <= 1.0])
        pos = np.concatenate(out)[:n] * np.array([case["sigma"], case["sigma"], 2 * case["sigma"]])
    else:
        pos = rng.normal(0.0, case["sigma"], (n, 3))
    mass = np.full(n, MASS * AMU)
    charge = np.ones(n, np.int32)
    if case["trap"] == "driven" and case["clouds"] == 1:
        mass[1::2] = 132.906 * AMU
    if case["trap"] == "paul":
        charge[::5] = 2
        charge[::17] = 3
    vel = rng.normal(0.0, 1.0, (n, 3)) * np.sqrt(KB * case["temp"] / mass)[:, None]
    return np.ascontiguousarray(pos), vel, mass, charge


def _fields(case):
    """Field parameters of every cloud, as dicts of the C struct's members."""
    if case["trap"] == "paul":
        f = {"flags": abi.SG_F_COULOMB | abi.SG_F_PAUL | abi.SG_F_TOF | abi.SG_F_FROZEN_T,
             "Vrf": 50.0, "Vdc": 5.0, "kappa": 0.001, "r0": 0.04, "z0": 0.04, "freq_rf": 50e5,
             "E_kick": 10.0}
        return [dict(f, coulomb_scale=1.0)]
    f = {"flags": abi.SG_F_COULOMB | abi.SG_F_PENNING, "coulomb_scale": 1.0, "B": 7.0, "V0": 10.0,
         "d0": 0.01, "r_el": 0.01}
    if case["trap"] != "driven":
        return [f]
    nu_c = E * 7.0 / (MASS * AMU) / (2 * PI)
    out = []
    for k in range(case["clouds"]):
        d = -5.0 + 10.0 * k / max(case["clouds"] - 1, 1)
        out.append(dict(f, flags=f["flags"] | abi.SG_F_QUAD | abi.SG_F_DIPOLE | abi.SG_F_FRICTION,
                        Uq=0.5, nu_q=nu_c + d, phi_q=0.0, tq_on=0.0, tq_off=1.0,
                        Ud=0.1, nu_d=2.3e3, phi_d=0.3, td_on=0.0, td_off=1.0, delta=1e3))
    return out


def _struct(f):
    p = abi.FieldParams()
    for k, v in f.items():
        setattr(p, k, v)
    return p


def _ode(case):
    o = abi.OdeParams()
    o.rtol, o.atol, o.h0, o.t0, o.t_end = 1e-9, 1e-15, case["h"], 0.0, 1.0
    o.adaptive, o.max_rejects, o.method = int(case["adaptive"]), 0, case["method"]
    return o


def _charges(case, seed):
    """positions, charges and per-ion factors of the Coulomb-only entry points."""
    rng = _rng(case, seed)
    pos = rng.normal(0.0, case["sigma"], (case["n"], 3))
    q = np.where(np.arange(case["n"]) % 5 == 0, 2.0, 1.0)
    return pos, q, KE * E * q * E / (MASS * AMU)


def _pair_sets(case, seed):
    rng = _rng(case, seed)
    xj = rng.normal(0.0, case["sigma"], (case["nj"], 3))
    # the reference's wrapper passes one array twice (bin/cunbody.cpp:43-90)
    same = case["ni"] == case["nj"]
    xi = xj.copy() if same else rng.normal(0.0, case["sigma"], (case["ni"], 3))
    mj = np.ones(case["nj"]) if same else rng.uniform(0.5, 2.0, case["nj"])
    return xj, mj, xi, float(np.float32(1e-23))


def _training(case, seed):
    rng = _rng(case, seed)
    n = case["n"]
    X = rng.normal(0.0, 0.5, (n, 16)).astype(np.float32)
    Y = (0.3 * X[:, 9] - 0.2 * X[:, 10] + 0.1 * X[:, 3] * X[:, 6]).astype(np.float32)
    P = 64 * 16 + 64 + 64 * 64 + 64 + 64 + 1
    w = np.zeros(P, np.float32)
    w[:1024] = rng.normal(0.0, 0.25, 1024)
    w[1088:5184] = rng.normal(0.0, 0.125, 4096)
    w[5248:5312] = rng.normal(0.0, 0.125, 64)
    return X, Y, w


# ---- the calls ---------------------------------------------------------------------
class _Integrate:
    def __init__(self, case, seed):
        self.pos, self.vel, mass, charge = _cloud(case, seed)
        self.k = case["attempts"]
        self.ctx = Context(0)
        fields = [_struct(f) for f in _fields(case)]
        self.batch = Batch(self.ctx, _counts(case), fields, [_ode(case)] * len(fields),
                           case["precision"])
        self.batch.upload(self.pos, self.vel, mass, charge)

    def run(self):
        if self.k:
            self.batch.attempts(self.k)
        else:
            self.batch.step()
        return self.batch.download()


class _Coupled(_Integrate):
    def run(self):
        self.batch.set_state(self.pos, self.vel)
        self.batch.step()
        return self.batch.download()


class _Force:
    def __init__(self, case, seed):
        self.args = _cloud(case, seed)
        self.fp = _struct(_fields(case)[0])
        self.prec = case["precision"]
        self.ctx = Context(0)

    def run(self):
        return self.ctx.force(*self.args, 3e-8, self.fp, self.prec)


class _Device:
    def __init__(self, case, seed):
        self.pos, self.q, self.kq = (torch.tensor(a, device="cuda") for a in _charges(case, seed))
        self.lib = abi.load()

    def run(self):
        acc = torch.empty_like(self.pos)
        abi.check(self.lib.sg_coulomb_accel_noalloc(
            len(self.q), self.pos.data_ptr(), self.q.data_ptr(), self.kq.data_ptr(),
            acc.data_ptr(), torch.cuda.current_stream().cuda_stream), "noalloc")
        return acc


class _Cunbody:
    def __init__(self, case, seed):
        self.xj, self.mj, self.xi, self.eps2 = _pair_sets(case, seed)
        self.lib = abi.load()

    def run(self):
        ai = np.zeros_like(self.xi)
        self.lib.cunbody1_force(abi.dptr(self.xj), abi.dptr(self.mj), abi.dptr(self.xi), self.eps2,
                                abi.dptr(ai), len(self.xi), len(self.xj))
        return ai


class _Train:
    def __init__(self, case, seed):
        self.X, self.Y, self.w = _training(case, seed)
        self.case = case
        self.ctx = Context(0)

    def run(self):
        return self.ctx.mlp_train(self.X, self.Y, self.w, iters=self.case["iters"],
                                  batch=self.case["batch"], lr=1e-3, seed=11)


_KINDS = {"integrate": _Integrate, "coupled": _Coupled, "force": _Force, "device": _Device,
          "cunbody": _Cunbody, "train": _Train}


def prepare(case, seed):
    return _KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


def _sums(case):
    """Coulomb sums a pass cannot do without: Dormand-Prince reuses one of its seven."""
    if case["kind"] in ("integrate", "coupled"):
        per = {5: 6, 4: 6, 1: 1}[case["method"]]
        # a new state needs the sum at its first stage too
        return per * max(case["attempts"], 1) + (1 if case["kind"] == "coupled" else 0)
    return 1


def work(case):
    """20 operations per ordered pair, the reference kernel's own tally
    (bin/nbody_kernel.cu:186-211)."""
    if case["kind"] == "train":
        p = 64 * 16 + 64 * 64 + 64
        return {"bytes": 4.0 * (17 * case["batch"] * case["iters"] + 8 * p),
                "flops": 6.0 * p * case["batch"] * case["iters"]}
    if case["kind"] == "cunbody":
        return {"bytes": 8.0 * (6 * case["ni"] + 4 * case["nj"]),
                "flops": 20.0 * case["ni"] * case["nj"]}
    if case["kind"] == "device":
        n = case["n"]
        return {"bytes": 64.0 * n, "flops": 20.0 * n * (n - 1)}
    counts = _counts(case)
    pairs = float(sum(c * (c - 1) for c in counts))
    # state in and out, mass and charge
    return {"bytes": 108.0 * sum(counts), "flops": 20.0 * pairs * _sums(case)}


# ---- the same in 64 bits, written out plainly ----------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pair_sum(xi, xj, q, self_pairs, eps2=0.0):
    """sum_j q_j (x_i - x_j) / (|x_i - x_j|^2 + eps2)^(3/2)."""
    out = torch.empty_like(xi)
    step = max(1, 32_000_000 // max(len(xj), 1))
    for a in range(0, len(xi), step):
        r = [xi[a:a + step, None, c] - xj[None, :, c] for c in range(3)]
        r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + eps2
        if self_pairs and not eps2:
            k = torch.arange(len(r2), device=r2.device)
            r2[k, a + k] = math.inf
        w = q / (r2 * r2.sqrt())
        for c in range(3):
            out[a:a + step, c] = (w * r[c]).sum(1)
    return out


def _accel(f, t, pos, vel, mass, q):
    fl, qm = f["flags"], (q * E / mass)[:, None]
    a = torch.zeros_like(pos)
    x, y, z = pos.unbind(1)
    if fl & abi.SG_F_PAUL:
        kv, c = f["kappa"] * f["Vdc"] / f["z0"] ** 2, math.cos(f["freq_rf"] * 2 * PI * t)
        c *= f["Vrf"] / f["r0"] ** 2
        a += qm * torch.stack([(kv - c) * x, (kv + c) * y, -2 * kv * z], 1)
    if fl & abi.SG_F_TOF:
        a[:, 0] += qm[:, 0] * f["E_kick"]
    if fl & abi.SG_F_PENNING:
        kp = f["V0"] / (2 * f["d0"] ** 2)
        a += qm * torch.stack([kp * x + f["B"] * vel[:, 1], kp * y - f["B"] * vel[:, 0],
                               -2 * kp * z], 1)
    if fl & abi.SG_F_QUAD:
        g = 2 * f["Uq"] / f["r_el"] ** 2 * math.cos(2 * PI * f["nu_q"] * t + f["phi_q"])
        a += qm * torch.stack([g * y, g * x, 0 * z], 1)
    if fl & abi.SG_F_DIPOLE:
        a[:, 0] += qm[:, 0] * f["Ud"] / f["r_el"] * math.cos(2 * PI * f["nu_d"] * t + f["phi_d"])
    if fl & abi.SG_F_FRICTION:
        a -= f["delta"] * vel
    k = (KE * E * q * E / mass)[:, None]
    return a + k * _pair_sum(pos, pos, q, True)


_DP = ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
        [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
        [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
        [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
       [0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1, 1],
       [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0.0],
       [71 / 57600, 0.0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40])
_CK = ([[], [0.2], [3 / 40, 9 / 40], [0.3, -0.9, 1.2], [-11 / 54, 2.5, -70 / 27, 35 / 27],
        [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]],
       [0, 0.2, 0.3, 0.6, 1.0, 0.875],
       [37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771], None)


def _advance(case, f, pos, vel, mass, q):
    a, c, b, e = _DP if case["method"] == 5 else _CK
    t, h, y, reject, errold = 0.0, case["h"], torch.cat([pos, vel], 1), False, 1e-4
    attempts, done = case["attempts"], 0
    while True:
        k = []
        for s in range(len(c)):
            ys = y + h * sum((w * kj for w, kj in zip(a[s], k)), torch.zeros_like(y))
            ts = t if f["flags"] & abi.SG_F_FROZEN_T else t + c[s] * h
            k.append(torch.cat([ys[:, 3:], _accel(f, ts, ys[:, :3], ys[:, 3:], mass, q)], 1))
        y5 = y + h * sum(w * kj for w, kj in zip(b, k))
        ok = True
        if case["adaptive"]:
            sk = 1e-15 + 1e-9 * torch.maximum(y.abs(), y5.abs())
            err = float(((h * sum(w * kj for w, kj in zip(e, k)) / sk) ** 2).mean().sqrt())
            ok = err <= 1.0
            scale = min(max(0.9 * err ** -0.2, 0.2), 10.0) if err else 10.0
            if not ok:
                h, reject = h * max(0.9 * err ** -0.2, 0.2), True
        if ok:
            y, t = y5, t + h
            if case["adaptive"]:
                h, reject, errold = h * (min(scale, 1.0) if reject else scale), False, err
        done += 1
        if done == attempts or (attempts == 0 and ok):
            return y[:, :3], y[:, 3:]


def _exact_train(case, seed):
    X, Y, w = (torch.tensor(v, dtype=torch.float64) for v in _training(case, seed))
    w, m, v, hist = w.clone(), torch.zeros_like(w), torch.zeros_like(w), []
    n, B, s, mask = case["n"], min(case["batch"], case["n"]), [11], (1 << 64) - 1

    def nxt():  # the seeded minibatch order of the training call
        s[0] = (s[0] + 0x9E3779B97F4A7C15) & mask
        z = s[0]
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return z ^ (z >> 31)

    perm, at = list(range(n)), n
    for it in range(case["iters"]):
        idx = []
        for _ in range(B):
            if at >= n:
                for i in range(n - 1, 0, -1):
                    j = nxt() % (i + 1)
                    perm[i], perm[j] = perm[j], perm[i]
                at = 0
            idx.append(perm[at])
            at += 1
        p = w.to(torch.float32).to(torch.bfloat16).to(torch.float64).requires_grad_()
        W1, b1, W2, b2 = p[:1024].view(64, 16), p[1024:1088], p[1088:5184].view(64, 64), p[5184:5248]
        h = torch.nn.functional.silu(X[idx] @ W1.T + b1)
        h = torch.nn.functional.silu(h @ W2.T + b2)
        loss = ((h @ p[5248:5312] + p[5312] - Y[idx]) ** 2).mean()
        (g,) = torch.autograd.grad(loss, p)
        hist.append(float(loss))
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** (it + 1))) / ((v / (1 - 0.999 ** (it + 1))).sqrt() + 1e-8)
    return w, torch.tensor(hist, dtype=torch.float64)


def exact(case, seed):
    d = _dev()
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "device":
        pos, q, kq = (torch.tensor(a, device=d) for a in _charges(case, seed))
        return kq[:, None] * _pair_sum(pos, pos, q, True)
    if case["kind"] == "cunbody":
        xj, mj, xi, eps2 = _pair_sets(case, seed)
        xj, mj, xi = (torch.tensor(a, device=d) for a in (xj, mj, xi))
        return -_pair_sum(xi, xj, mj, False, eps2).cpu().numpy()
    counts = _counts(case)
    if sum(c * c for c in counts) * float(_sums(case)) > 4e10 or case.get("method") == 1:
        return None  # more than about 20 seconds; Gear starts from constants of its own
    pos, vel, mass, charge = (torch.tensor(a, device=d) for a in _cloud(case, seed))
    charge = charge.to(torch.float64)
    if case["kind"] == "force":
        return _accel(_fields(case)[0], 3e-8, pos, vel, mass, charge).cpu().numpy()
    out, at = [], 0
    for n, f in zip(counts, _fields(case)):
        s = slice(at, at + n)
        out.append(_advance(case, f, pos[s], vel[s], mass[s], charge[s]))
        at += n
    return tuple(torch.cat(v).cpu().numpy() for v in zip(*out))

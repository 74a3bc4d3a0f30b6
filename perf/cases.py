"""The measured work of this repository: particle-to-particle evaluations as a vortex-particle
program asks for them, through the public entry points (the drop-in hooks, the device context,
the autograd functions and the device-resident step).

A case is a dict of plain values:

  kind     what is called:
             hook   `pfield.UJ(pfield, ...)` on the host 46-row particle matrix (the drop-in)
             uj     `Context.uj_dev` on device arrays
             grad   `autodiff.uj` (and `autodiff.estr` with sfs) forward and backward
             estr   `Context.estr_dev`, the SFS stretching pass
             dyn    `Context.dynamic_diff_dev`, the dynamic procedure's test-filter differences
             near   `Context.p2p_leaflist_dev`, the near field over octree leaf pairs
             step   `device_step.rk3_step` with core spreading and relaxation
  field    the particle set: cloud (uniform, random strengths), ring (one vortex ring),
           rings (two leapfrogging rings), jet (a cylinder of solenoidal vorticity)
  n        particles; kernel 0..3 (singular, Gaussian, Gaussian-erf, Winckelmans)
  mixed    False: FP64; True: FP32 pair arithmetic with FP64 block sums

The mixed form's sums are FP32-accurate numbers in FP64 arrays; run() hands them over as
float32, the type that holds what they carry.  The FP64 form's outputs stay float64.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "flowvpm.jl_gb300"))
import vpm_gb300 as vpm                                     # noqa: E402
from vpm_gb300 import autodiff, device_step, workloads      # noqa: E402

F64 = torch.float64
ALPHA = 0.999          # the two-level dynamic procedure's filter ratio
LEAF, THETA = 64, 0.4  # octree leaf size and acceptance criterion of the near-field workload
NU, DT = 1e-3, 1e-3    # core spreading's viscosity and the time step of the step cases


def listed():
    return [
        # the smallest drop-in call: the isolated ring of the reference's ring test (200 sections of 7),
        # a UJ with its SFS pass on the host matrix in the default precision
        dict(name="hook_ring_1400_f64", kind="hook", field="ring", n=1400, kernel=2, mixed=False, sfs=True),
        # an ordinary drop-in call of a program that selects the mixed form; odd size
        dict(name="hook_cloud_150k_mixed", kind="hook", field="cloud", n=150_001, kernel=2, mixed=True, sfs=False),
        # a small field on the device, as in the first steps of a run: launches and latency count
        dict(name="uj_cloud_4k_mixed", kind="uj", field="cloud", n=4099, kernel=2, mixed=True, sfs=False),
        # the random cloud at the benchmark's size
        dict(name="uj_cloud_1m_mixed", kind="uj", field="cloud", n=1 << 20, kernel=2, mixed=True, sfs=False),
        # the algebraic kernel of the reference's ring test, at an ordinary odd size
        dict(name="uj_cloud_50k_winck_mixed", kind="uj", field="cloud", n=50_001, kernel=3, mixed=True, sfs=False),
        # the default precision at the cloud workload's lower end
        dict(name="uj_cloud_16k_f64", kind="uj", field="cloud", n=16_411, kernel=2, mixed=False, sfs=False),
        # the ring of the rollout-gradient workload: value and gradient of one evaluation
        dict(name="grad_ring_32k_mixed", kind="grad", field="ring", n=32_000, kernel=2, mixed=True, sfs=False),
        # the same in the default precision with the SFS pass, at a size such rollouts are checked at
        dict(name="grad_ring_5k_sfs_f64", kind="grad", field="ring", n=5_600, kernel=2, mixed=False, sfs=True),
        # the stretching pass and the dynamic procedure's differences on the leapfrogging rings
        dict(name="estr_rings_200k_mixed", kind="estr", field="rings", n=200_000, kernel=2, mixed=True, sfs=False),
        dict(name="dyn_rings_100k_mixed", kind="dyn", field="rings", n=100_000, kernel=2, mixed=True, sfs=False),
        # the jet cloud's near field: list build, UJ and SFS over the leaf pairs
        dict(name="near_jet_1m_mixed", kind="near", field="jet", n=1 << 20, kernel=2, mixed=True, sfs=True),
        # one whole time step of the rings (four evaluations and the per-particle work)
        dict(name="step_rings_60k_mixed", kind="step", field="rings", n=60_000, kernel=2, mixed=True, sfs=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hook", "uj", "uj", "uj", "grad", "estr", "dyn", "near", "step"])
    mixed = rng.random() < 0.7
    kernel = rng.choice([2, 2, 2, 3, 1, 0])
    if kind == "hook":
        n = _log(rng, 1_000, 250_000 if mixed else 20_000)
        return dict(kind=kind, field=rng.choice(["ring", "cloud"]), n=n, kernel=rng.choice([2, 3]), mixed=mixed,
                    sfs=rng.random() < 0.5)
    if kind == "uj":
        n = _log(rng, 2_000, 600_000 if mixed else 40_000)
        return dict(kind=kind, field=rng.choice(["cloud", "cloud", "rings", "jet"]), n=n, kernel=kernel, mixed=mixed,
                    sfs=False)
    if kind == "grad":
        n = _log(rng, 1_400, 60_000 if mixed else 8_000)
        return dict(kind=kind, field="ring", n=n, kernel=rng.choice([2, 2, 3]), mixed=mixed, sfs=rng.random() < 0.5)
    if kind in ("estr", "dyn"):   # the FP64 step takes the differences as two evaluations, not as this call
        mixed = mixed or kind == "dyn"
        n = _log(rng, 10_000, 250_000 if mixed else 20_000)
        return dict(kind=kind, field="rings", n=n, kernel=2, mixed=mixed, sfs=False)
    if kind == "near":
        n = _log(rng, 20_000, 1_048_576 if mixed else 200_000)
        return dict(kind=kind, field="jet", n=n, kernel=2, mixed=mixed, sfs=rng.random() < 0.6)
    return dict(kind=kind, field="rings", n=_log(rng, 10_000, 150_000), kernel=2, mixed=True, sfs=False)


# ------------------------------------------------------------------ particle sets
def _fit(X, G, s, n):
    return X[:n], G[:n], s[:n]


def _field(case, seed):
    """x[n,3], gamma[n,3], sigma[n] on the GPU.  Rings are advected fields in earnest, so their
    particles sit a little off the generator's regular places, by the seed."""
    n, f = int(case["n"]), case["field"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    u = lambda *sh: torch.rand(*sh, generator=gen, device="cuda", dtype=F64)     # noqa: E731
    g = lambda *sh: torch.randn(*sh, generator=gen, device="cuda", dtype=F64)    # noqa: E731
    if f == "cloud":
        return u(n, 3), 1e-3 * g(n, 3), 0.01 + 0.02 * u(n)
    if f == "jet":
        r, th = 0.5 * u(n).sqrt(), 2 * math.pi * u(n)
        x = torch.stack([r * th.cos(), r * th.sin(), 4.0 * u(n)], 1)
        k, a, phi = 8.0 * g(64, 3), g(64, 3) / 8.0, 2 * math.pi * u(64)
        om = -torch.sin(x @ k.T + phi) @ torch.linalg.cross(k, a)
        # the core size keeps the million-particle cloud's overlap at every n
        return x, (math.pi / n) * om, torch.full((n,), 0.02 * ((1 << 20) / n) ** (1 / 3), device="cuda", dtype=F64)
    if f == "ring":
        nper = 7 if n <= 8_000 else 32
        X, G, s = workloads.rollout_ring(-(-n // nper), nper)
    else:
        X, G, s = workloads.leapfrog_rings(2 * 10 * -(-n // 20), 10)
    X, G, s = (torch.tensor(v, device="cuda") for v in _fit(X, G, s, n))
    x = X + 2e-3 * g(n, 3)
    return x, G * (1 + 0.02 * g(n, 1)), s * (1 + 0.02 * (u(n) - 0.5))


def _gradients(x, gam, sig):
    """A smooth velocity gradient, J[n,9], as a UJ evaluation of the rings leaves it."""
    p = torch.stack([torch.sin(3 * x[:, 0] + x[:, 1]), torch.cos(2 * x[:, 1] - x[:, 2]),
                     torch.sin(x[:, 2] + 4 * x[:, 0]), x[:, 0] * x[:, 1], torch.cos(5 * x[:, 2]),
                     x[:, 1] - x[:, 2], torch.sin(2 * x[:, 0]) * x[:, 2], torch.cos(x[:, 0] + x[:, 1]),
                     torch.sin(x[:, 1] * 3)], 1)
    return p.contiguous()


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind, n = case["kind"], int(case["n"])
    prec = vpm.FP32COMP if case["mixed"] else vpm.FP64
    s = dict(kind=kind, kernel=int(case["kernel"]), prec=prec, sfs=bool(case["sfs"]), mixed=bool(case["mixed"]))
    x, gam, sig = _field(case, seed)
    if kind == "hook":
        k = {2: vpm.gaussianerf, 3: vpm.winckelmans}[s["kernel"]]
        pf = vpm.ParticleField(n, kernel=k, UJ=vpm.UJ_gb300_mixed if case["mixed"] else vpm.UJ_gb300)
        pf.add_particles(x.cpu().numpy(), gam.cpu().numpy(), sig.cpu().numpy())
        s["pf"] = pf
        return s
    s.update(x=x, gam=gam, sig=sig, ctx=vpm.default_context())
    if kind == "grad":
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        s["Ub"] = torch.randn(n, 3, generator=gen, device="cuda", dtype=F64)
        s["Jb"] = torch.randn(n, 9, generator=gen, device="cuda", dtype=F64)
        s["Sb"] = torch.randn(n, 3, generator=gen, device="cuda", dtype=F64)
    if kind in ("estr", "dyn"):
        s["J"] = _gradients(x, gam, sig)
    return s


def _as(s, *v):
    return [t.to(torch.float32) for t in v] if s["mixed"] else list(v)


def run(s):
    kind, kernel, prec = s["kind"], s["kernel"], s["prec"]
    if kind == "hook":
        pf = s["pf"]
        pf.UJ(pf, sfs=s["sfs"], reset=True, reset_sfs=s["sfs"])
        t = np.float32 if s["mixed"] else np.float64
        out = [pf.U.astype(t), pf.J.astype(t)]
        return out + [pf.SFS_values.astype(t)] if s["sfs"] else out
    ctx, x, gam, sig = s["ctx"], s["x"], s["gam"], s["sig"]
    n = x.shape[0]
    new = lambda c: torch.zeros(n, c, device="cuda", dtype=F64)      # noqa: E731
    if kind == "uj":
        U, J = new(3), new(9)
        ctx.uj_dev(x, x, gam, sig, U, J, kernel, prec)
        return _as(s, U, J)
    if kind == "grad":
        xr, gr, sr = (t.detach().requires_grad_() for t in (x, gam, sig))
        U, J = autodiff.uj(xr, gr, sr, kernel, prec, ctx)
        outs, bars = [U, J], [s["Ub"], s["Jb"]]
        if s["sfs"]:
            outs.append(autodiff.estr(xr, gr, sr, J, kernel, prec, True, ctx))
            bars.append(s["Sb"])
        grads = torch.autograd.grad(outs, (xr, gr, sr), bars)
        return _as(s, *[o.detach() for o in outs], *grads)
    if kind == "estr":
        S = new(3)
        ctx.estr_dev(x, s["J"], x, gam, sig, s["J"], S, kernel, prec)
        return _as(s, S)
    if kind == "dyn":
        dJ, dS = new(9), new(3)
        ctx.dynamic_diff_dev(x, gam, sig, s["J"], ALPHA, dJ, dS, kernel, prec)
        return _as(s, dJ, dS)
    if kind == "near":
        U, J, S = new(3), new(9), new(3)
        ctx.p2p_leaflist_dev(x, gam, sig, U, J, S if s["sfs"] else None, leaf_size=LEAF, theta=THETA, kernel=kernel,
                             precision=prec, sfs=s["sfs"])
        return _as(s, U, J, S) if s["sfs"] else _as(s, U, J)
    # the step works in place: a program's own state, here a copy so that a pass can be repeated
    fld = device_step.DeviceField(x.clone(), gam.clone(), sig.clone(), kernel=kernel, precision=prec)
    device_step.rk3_step(fld, DT, ctx, viscous=device_step.CoreSpreadingParams(nu=NU, sgm0=0.05), relax_rlxf=0.3)
    return _as(s, fld.x, fld.gam, fld.sig, fld.U, fld.J)


def work(case):
    n, kind = int(case["n"]), case["kind"]
    pairs = float(n) * n
    if kind in ("hook", "uj"):
        return {"bytes": n * (56 + 96 + (24 if case["sfs"] else 0)), "flops": (74 + (25 if case["sfs"] else 0)) * pairs}
    if kind == "grad":
        return {"bytes": n * (56 + 2 * 96 + 56 + (48 if case["sfs"] else 0)),
                "flops": (74 + 186 + (75 if case["sfs"] else 0)) * pairs}
    if kind == "estr":
        return {"bytes": n * (56 + 72 + 24), "flops": 25 * pairs}
    if kind == "dyn":
        return {"bytes": n * (56 + 72 + 96), "flops": 2 * (74 + 25) * pairs}
    if kind == "near":   # about 2,470 near particles for each at this leaf size and criterion
        near = 2470.0 * n if n > 4000 else pairs
        return {"bytes": n * (56 + 120), "flops": (74 + (25 if case["sfs"] else 0)) * near}
    return {"bytes": n * (2 * 56 + 96), "flops": 4 * 74 * pairs}


# ------------------------------------------------------------------ 64-bit values
C4 = 1 / (4 * math.pi)
_CHUNK = 1 << 24   # pairs evaluated at once


def _df(k):   # (2m+1)!!
    return math.prod(range(1, 2 * k + 2, 2))


def _GQ(kernel, s):
    """G = g/rho^3 and Q = (3 g - rho g')/(3 rho^5) as functions of s = rho^2 > 0, without the
    cancellation at small rho of the kernels' literal form."""
    if kernel == 0:
        r = s.rsqrt()
        return r ** 3, r ** 5
    if kernel == 3:
        return (s + 2.5) * (s + 1) ** -2.5, (s + 3.5) * (s + 1) ** -3.5
    rho = s.sqrt()
    if kernel == 1:
        t = rho ** 3
        e = torch.exp(-t)
        small = t < 0.5
        ts = torch.where(small, t, torch.full_like(t, 0.1))
        q = sum((-1) ** m * (m + 1) / math.factorial(m + 2) * ts ** m for m in range(18))   # (1 - e - t e)/t^2
        tb = torch.where(small, torch.ones_like(t), t)
        eb = torch.exp(-tb)
        return -torch.expm1(-t) / t, torch.where(small, q, (1 - eb - tb * eb) / tb ** 2) * rho
    # Gaussian-erf: Kummer's series of erf below s = 2
    c2, e = math.sqrt(2 / math.pi), torch.exp(-0.5 * s)
    ss = torch.clamp(s, max=2.0)
    S2 = torch.zeros_like(s)
    for m in reversed(range(26)):
        S2 = S2 * ss + 1.0 / _df(m + 2)
    big = s > 2.0
    sb = torch.where(big, s, torch.full_like(s, 3.0))
    rb, eb = sb.sqrt(), torch.exp(-0.5 * sb)
    Gb = (torch.erf(rb / math.sqrt(2)) - c2 * rb * eb) / rb ** 3
    return torch.where(big, Gb, c2 * e * (1 / 3 + s * S2)), torch.where(big, (Gb - c2 * eb / 3) / sb, c2 * e * S2)


def _zeta(kernel, s):
    if kernel == 0:
        return (s == 0).to(F64)
    if kernel == 1:
        return 3 * C4 * torch.exp(-s * s.sqrt())
    if kernel == 2:
        return torch.exp(-0.5 * s) / (2 * math.pi) ** 1.5
    return 7.5 * C4 * (s + 1) ** -3.5


def _uj_rows(kernel, xt, x, gam, sig):
    """U[t,3], J[t,9] of targets xt from all sources (pairs at r = 0 skipped)."""
    d = xt[:, None, :] - x[None, :, :]
    dx, dy, dz = d.unbind(-1)
    r2 = dx * dx + dy * dy + dz * dz
    sg = torch.ones_like(sig) if kernel == 0 else sig
    r2 = torch.where(r2 == 0, sg * sg, r2)     # c = 0 there; the Kronecker term is taken out below
    on = ((dx != 0) | (dy != 0) | (dz != 0)).to(F64)
    G, Q = _GQ(kernel, r2 / (sg * sg))
    A = -C4 * on * G / sg ** 3
    B = 3 * C4 * on * Q / sg ** 5
    gx, gy, gz = gam.unbind(-1)
    c = (dy * gz - dz * gy, dz * gx - dx * gz, dx * gy - dy * gx)
    U = [(A * v).sum(1) for v in c]
    W = [A @ v for v in (gx, gy, gz)]
    J = [[(B * c[k] * dl).sum(1) for k in range(3)] for dl in (dx, dy, dz)]     # J[l][k] = dU_k/dx_l
    J[0][1] = J[0][1] - W[2]
    J[0][2] = J[0][2] + W[1]
    J[1][0] = J[1][0] + W[2]
    J[1][2] = J[1][2] - W[0]
    J[2][0] = J[2][0] - W[1]
    J[2][1] = J[2][1] + W[0]
    return torch.stack(U, 1), torch.stack([J[l][k] for l in range(3) for k in range(3)], 1)


def _estr_rows(kernel, xt, Jt, x, gam, sig, J):
    """SFS[t,3] of the transposed scheme: sum zeta (J_t - J_s)^T Gamma_s."""
    d = xt[:, None, :] - x[None, :, :]
    z = _zeta(kernel, (d * d).sum(-1) / (sig * sig)) / sig ** 3
    v = (J.view(-1, 3, 3) * gam[:, None, :]).sum(2)         # J_s^T Gamma_s
    zg = z @ gam
    return (Jt.view(-1, 3, 3) * zg[:, None, :]).sum(2) - z @ v


def _rows(n):
    step = max(1, _CHUNK // n)
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _uj(kernel, x, gam, sig):
    p = [_uj_rows(kernel, x[a:b], x, gam, sig) for a, b in _rows(x.shape[0])]
    return torch.cat([v[0] for v in p]), torch.cat([v[1] for v in p])


def _estr(kernel, x, gam, sig, J):
    return torch.cat([_estr_rows(kernel, x[a:b], J[a:b], x, gam, sig, J) for a, b in _rows(x.shape[0])])


def _exact_grad(kernel, sfs, x, gam, sig, Ub, Jb, Sb):
    U, J = _uj(kernel, x, gam, sig)
    gx, gg, gs, gJ = torch.zeros_like(x), torch.zeros_like(gam), torch.zeros_like(sig), Jb.clone()
    S = _estr(kernel, x, gam, sig, J) if sfs else None
    leaves = [t.detach().requires_grad_() for t in (x, gam, sig)]
    if sfs:
        Jr = J.detach().requires_grad_()
        for a, b in _rows(x.shape[0] * 4):
            if a >= x.shape[0]:
                break
            b = min(b, x.shape[0])
            L = (_estr_rows(kernel, leaves[0][a:b], Jr[a:b], *leaves, Jr) * Sb[a:b]).sum()
            p = torch.autograd.grad(L, (*leaves, Jr))
            gx, gg, gs, gJ = gx + p[0], gg + p[1], gs + p[2], gJ + p[3]
    step = max(1, _CHUNK // (2 * x.shape[0]))
    for a in range(0, x.shape[0], step):
        b = min(x.shape[0], a + step)
        u, j = _uj_rows(kernel, leaves[0][a:b], *leaves)
        p = torch.autograd.grad((u * Ub[a:b]).sum() + (j * gJ[a:b]).sum(), leaves)
        gx, gg, gs = gx + p[0], gg + p[1], gs + p[2]
    return [U, J] + ([S] if sfs else []) + [gx, gg, gs]


def _exact_step(kernel, x, gam, sig):
    """rVPM (f = 0, g = 1/5) low-storage RK3 with core spreading, then Pedrizzetti relaxation."""
    M0, M3, M8, M7 = (torch.zeros_like(t) for t in (x, gam, sig, sig))
    for a, b in ((0.0, 1 / 3), (-5 / 9, 15 / 16), (-153 / 128, 8 / 15)):
        U, J = _uj(kernel, x, gam, sig)
        S = (J.view(-1, 3, 3) * gam[:, None, :]).sum(2)
        Z = 0.2 * (S * gam).sum(1) / (gam * gam).sum(1)
        M0 = a * M0 + DT * U
        M3 = a * M3 + DT * (S - 3 * Z[:, None] * gam)
        M8 = a * M8 - DT * sig * Z
        x, gam, sig = x + b * M0, gam + b * M3, sig + b * M8
        M7 = a * M7 + DT * 2 * NU
        sig = (sig * sig + b * M7).sqrt()
    U, J = _uj(kernel, x, gam, sig)
    w = torch.stack([J[:, 5] - J[:, 7], J[:, 6] - J[:, 2], J[:, 1] - J[:, 3]], 1)
    gam = 0.7 * gam + 0.3 * gam.norm(dim=1, keepdim=True) / w.norm(dim=1, keepdim=True) * w
    return [x, gam, sig, U, J]


def exact(case, seed):
    n, kind, kernel = int(case["n"]), case["kind"], int(case["kernel"])
    # past these sizes plain torch takes too long; the near field's value depends on the octree's
    # leaf pairs, whose construction in plain torch takes too long too
    most = {"hook": 200_000, "uj": 200_000, "grad": 40_000, "estr": 250_000, "dyn": 130_000, "near": 0, "step": 100_000}
    if n > most[kind]:
        return None
    x, gam, sig = _field(case, seed)
    with torch.no_grad():
        if kind in ("hook", "uj"):
            U, J = _uj(kernel, x, gam, sig)
            return [U, J] + ([_estr(kernel, x, gam, sig, J)] if case["sfs"] else [])
        if kind == "estr":
            return [_estr(kernel, x, gam, sig, _gradients(x, gam, sig))]
        if kind == "dyn":
            J = _gradients(x, gam, sig)
            dJ = _uj(kernel, x, gam, ALPHA * sig)[1] - _uj(kernel, x, gam, sig)[1]
            return [dJ, _estr(kernel, x, gam, ALPHA * sig, J + dJ) - _estr(kernel, x, gam, sig, J)]
        if kind == "step":
            return _exact_step(kernel, x, gam, sig)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    b = [torch.randn(n, c, generator=gen, device="cuda", dtype=F64) for c in (3, 9, 3)]
    return _exact_grad(kernel, bool(case["sfs"]), x, gam, sig, *b)

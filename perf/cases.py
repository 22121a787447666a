"""The work a user has this framework do, as cases that can be timed and compared.

Every case goes through the public entry points of lydion_b200 (M1Context, M1Batch). The kinds:

  run      a stretch of a static-cloud run: the state of a restart file goes up, `steps` driver
           iterations run, the step records and the state at the save point come back
  batch    the same for many small clouds of uneven size held in one context
  adjoint  the gradients of M_F and the edge spectrum through `steps` iterations
  host     one iteration on a state the program keeps in host memory, updated in place
  phases   the driver loop written out in the reference's calls, state resident on the device
  rhd      a radiation-hydrodynamics sub-cycle: opacities from the gas, two absorption
           sub-steps, the transport step
  bands    a few broad bands advected with their own opacities (no line transfer)

Sizes are those of lydion_b200/workloads.py and bench.py, or odd ones in between. The states have
the spectra of evolved runs: flat across the optically thick core, cut off a few (a tau)^(1/3)
out, so that FindActiveBins leaves out the far wings as it does in a run.
"""
import math

import numpy as np
import torch

from lydion_b200 import constants as K
from lydion_b200 import m1
from lydion_b200 import workloads as W

PREC = {"fp64": 0, "mixed": 1, "fp32": 2}
FIELDS = ("J", "H_r", "H_Z")


def listed():
    return [
        # a parity-size cloud: latency and launches are all there is
        dict(name="run_tiny", kind="run", nr=24, nz=20, nnu=16, steps=20, prec="fp64", flux="glf", bottom="reflect",
             tau0=1e5, umax=150.0, rs=0.5),
        # the plain point-source cloud of the static tests
        dict(name="run_point_64", kind="run", nr=64, nz=64, nnu=64, steps=50, prec="fp64", flux="glf",
             bottom="reflect", tau0=1e6, umax=0.0, rs=0.0),
        # the dusty outflowing cloud of the benchmark, in its three precision forms
        dict(name="run_256_fp64", kind="run", nr=256, nz=256, nnu=64, steps=24, prec="fp64", flux="glf",
             bottom="reflect", tau0=1e8, umax=200.0, rs=0.5),
        dict(name="run_256_mixed", kind="run", nr=256, nz=256, nnu=64, steps=24, prec="mixed", flux="glf",
             bottom="reflect", tau0=1e8, umax=200.0, rs=0.5),
        dict(name="run_256_fp32", kind="run", nr=256, nz=256, nnu=64, steps=24, prec="fp32", flux="glf",
             bottom="reflect", tau0=1e8, umax=200.0, rs=0.5),
        # odd sizes, the HLL flux and an open bottom
        dict(name="run_ragged_hll", kind="run", nr=131, nz=203, nnu=50, steps=30, prec="fp64", flux="hll",
             bottom="outflow", tau0=1e7, umax=60.0, rs=0.5),
        # a large field with 128 bins
        dict(name="run_large", kind="run", nr=512, nz=512, nnu=128, steps=6, prec="fp64", flux="glf",
             bottom="reflect", tau0=1e7, umax=30.0, rs=0.2),
        # a parameter sweep: small clouds of uneven size advancing together
        dict(name="batch_24", kind="batch", clouds=24, side_max=96, nnu=48, steps=40, prec="fp64"),
        # gradients through a turbulent-size cloud, every step kept
        dict(name="adjoint_128", kind="adjoint", nr=128, nz=128, nnu=48, steps=20, flux="glf", every=1, tau0=3e7,
             umax=50.0, rs=0.5),
        # a host program that owns its state and hands it over every step
        dict(name="host_256", kind="host", nr=256, nz=256, nnu=64, prec="fp64", flux="glf", bottom="reflect",
             tau0=1e8, umax=200.0, rs=0.5),
        # the Lyman-alpha part of a radiation-hydrodynamics sub-cycle
        dict(name="rhd_192", kind="rhd", nr=192, nz=192, nnu=64, prec="fp64"),
        # stellar and infrared bands beside the line
        dict(name="bands_256", kind="bands", nr=256, nz=256, nnu=8, steps=10, prec="fp64", flux="glf"),
    ]


def draw(rng):
    """One more case of the ranges above: sides 12..400, 8..128 bins, all precision forms, fluxes and
    boundaries, from a few hundred cells to the size of the large field."""
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "run", "batch", "adjoint", "host", "phases", "rhd", "bands"])
    c = dict(kind=kind, prec=rng.choice(["fp64", "fp64", "mixed", "fp32"]))
    if kind == "batch":
        c.update(clouds=rng.randint(5, 28), side_max=rng.choice([48, 64, 80, 96]), nnu=rng.choice([24, 32, 48, 64]),
                 steps=rng.randint(8, 40))
        return c
    c.update(nr=side(12, 400), nz=side(12, 400), nnu=2 * rng.randint(8, 32) if rng.random() < 0.7 else
             2 * rng.randint(33, 64))
    c.update(flux=rng.choice(["glf", "glf", "hll"]), bottom=rng.choice(["reflect", "reflect", "outflow"]),
             tau0=float("%.3g" % 10.0 ** rng.uniform(4.0, 8.0)), umax=float(rng.choice([0, 30, 100, 200])),
             rs=rng.choice([0.0, 0.2, 0.5]))
    size = c["nr"] * c["nz"] * c["nnu"]
    c["steps"] = max(2, min(50, int(1.5e8 / size), rng.randint(6, 50)))
    if kind == "adjoint":
        c["nr"], c["nz"], c["nnu"] = min(c["nr"], 160), min(c["nz"], 160), min(c["nnu"], 64)
        c["steps"] = min(c["steps"], 20)
        c["every"] = rng.choice([1, 1, 5, -1])
        del c["bottom"]
        c["prec"] = "fp64"
    elif kind == "host":
        c["prec"] = "fp64"
        c["nz"] = max(c["nz"], 24)
        del c["steps"]
    elif kind == "rhd":
        c["prec"] = "fp64"
        for k in ("flux", "bottom", "tau0", "umax", "rs", "steps"):
            del c[k]
    elif kind == "bands":
        c["nnu"] = 2 * rng.randint(2, 10)
        c["steps"] = min(c["steps"], 12)
        for k in ("bottom", "tau0", "umax", "rs"):
            del c[k]
    elif kind == "phases":
        c["steps"] = min(c["steps"], 12)
    return c


def work(case):
    """Bytes: state and H_voigt read once and the state written once per iteration, per-cell inputs;
    operations: about 700 per cell and bin of an iteration (two faces, closure, factors, solve)."""
    e = 4 if case.get("prec") == "fp32" else 8
    n = case["clouds"] * (0.6 * case["side_max"]) ** 2 if case["kind"] == "batch" else case["nr"] * case["nz"]
    cb = n * case["nnu"]
    k = case["kind"]
    if k == "adjoint":
        # forward, reverse of the frequency step and of the advection
        return {"bytes": case["steps"] * cb * 8 * (7 + 11 + 11), "flops": case["steps"] * cb * 2500}
    if k == "bands":
        return {"bytes": case["steps"] * cb * e * 7, "flops": case["steps"] * cb * 450}
    if k == "host":
        return {"bytes": cb * 8 * 7 + n * 160, "flops": cb * 700}
    if k == "rhd":
        return {"bytes": cb * 8 * (3 * 7 + 1) + n * 400, "flops": cb * 800}
    return {"bytes": case["steps"] * (cb * e * 7 + n * 160), "flops": case["steps"] * cb * 700}


# ---- inputs -----------------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _voigt(T, freq):
    """A line profile H(a, x) on (cells, bins): Doppler core and damping wings."""
    T = torch.as_tensor(T, dtype=torch.float64, device=_device()).reshape(-1, 1)
    b = K.b_prefact * torch.sqrt(T)
    x = torch.as_tensor(freq.nuC - K.nu_lya, device=T.device)[None, :] / (b * (K.nu_lya / K.c))
    a = K.a_prefact / b
    return torch.exp(-x * x) + a / math.sqrt(math.pi) / (x * x + 1.5) * (1.0 - torch.exp(-x * x) * 0.9)


def _state(cloud, gen, amp):
    """J and H of an evolved run: radially falling, outward fluxes, a spectrum that is flat across the
    thick core and ends a few (a tau)^(1/3) out, shifted and widened by the outflow."""
    dev = _device()
    f = cloud.freq
    T0 = float(np.asarray(cloud.T).flat[0])
    x = torch.as_tensor((f.nuC - K.nu_lya) / K.compute_dnuD(T0), device=dev)
    at = max(1.0, K.compute_a(T0) * cloud.tau0)
    v = float(np.hypot(cloud.u_r, cloud.u_Z).max()) / K.compute_b(T0)
    xw = 1.0 + at ** (1.0 / 3.0) + 0.5 * v
    s = torch.exp(-torch.clamp(((x + 0.4 * v) / xw).abs() ** 3, max=120.0))
    r = torch.as_tensor(cloud.geom.rCoM, device=dev)[None, :, None] / K.pc
    z = (torch.as_tensor(cloud.geom.ZCoM, device=dev) - cloud.z_center)[:, None, None] / K.pc
    R = torch.sqrt(r * r + z * z) + 1e-3
    n = torch.rand((3, cloud.nz, cloud.nr, f.n_nu), generator=gen, device=dev, dtype=torch.float64)
    J = amp * s * torch.exp(-3.0 * R * R) * (0.95 + 0.1 * n[0])
    fl = (0.02 + 0.7 * R * R / (1.0 + R * R)) * (1.0 - 0.8 * torch.exp(-(x / xw) ** 2)) * (0.9 + 0.2 * n[1])
    th = 0.3 * (n[2] - 0.5)
    J = torch.clamp(J, min=1e-60)
    return J, J * fl * (r / R * torch.cos(th) - z / R * torch.sin(th)), \
        J * fl * (z / R * torch.cos(th) + r / R * torch.sin(th))


def _pinned(t):
    a = m1.pinned_zeros(tuple(t.shape))
    torch.from_numpy(a).copy_(t)
    return a


def _rng(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(1000003 * (seed + 1))
    return g, np.random.default_rng(seed)


def _cloud(case, rng, **over):
    c = dict(case, **over)
    cl = W.static_cloud(c["nr"], c["nz"], c["nnu"], tau0=c.get("tau0", 1e6) * rng.uniform(0.8, 1.25),
                        T0=c.get("T0", 1e4), tau_abs=c.get("tau_abs", 1.0), rs=c.get("rs", 0.5),
                        umax_kms=c.get("umax", 0.0), pd0=c.get("pd0", 1e-7),
                        bc_z_bot=W.BC_OUTFLOW if c.get("bottom") == "outflow" else W.BC_REFLECT,
                        flux_method=W.FLUX_HLL if c.get("flux") == "hll" else W.FLUX_GLF, freq=c.get("freq"))
    g = cl.geom
    if c["kind"] == "adjoint":
        # thin gas around the cloud: with none the gradients in its opacity are 0 / 0
        cl.alpha = np.maximum(cl.alpha, 1e-5 * cl.alpha.max())
    w = rng.uniform(0.7, 1.4, size=cl.alpha.shape)          # clumps
    cl.alpha, cl.alpha_c = cl.alpha * w, cl.alpha_c * w
    if c.get("umax", 0.0) > 0:
        s = rng.normal(size=cl.alpha.shape) * 1e5 / g.r[-1]  # a little shear on the outflow
        cl.dur_dZ, cl.duZ_dr = s, -0.5 * s
    return cl


def _inputs(case, seed):
    """Everything a single-cloud case feeds the framework: the cloud, its line profile and the state."""
    gen, rng = _rng(seed)
    kind = case["kind"]
    cl = _cloud(case, rng, **(dict(tau0=1e7, umax=100.0) if kind == "rhd" else {}))
    hv = _voigt(cl.T, cl.freq).reshape(cl.nz, cl.nr, cl.n_nu)
    return cl, hv, _state(cl, gen, 1e-12), gen, rng


def _batch_clouds(case, seed):
    _, rng = _rng(seed)
    sides = [s for s in W.C3_SIDES if s <= case["side_max"]] + [17, 39]
    first = _cloud(dict(kind="batch", nr=16, nz=16, nnu=case["nnu"]), rng)
    out = []
    shape = np.random.default_rng(7)                        # the sizes belong to the case, not to the seed
    for _ in range(case["clouds"]):
        nr, nz = int(shape.choice(sides)), int(shape.choice(sides))
        out.append(_cloud(dict(kind="batch", nr=nr, nz=nz, nnu=case["nnu"], tau0=10.0 ** rng.uniform(4, 8), tau_abs=rng.uniform(0, 2),
                               T0=10.0 ** rng.uniform(2, 4), umax=rng.uniform(0, 100), freq=first.freq), rng))
    return out


# ---- one pass ---------------------------------------------------------------------------------

def prepare(case, seed):
    kind, prec = case["kind"], PREC[case.get("prec", "fp64")]
    s = {"case": case, "kind": kind}
    if kind == "batch":
        clouds = _batch_clouds(case, seed)
        gen, _ = _rng(seed)
        ctx = m1.batch_for_clouds(clouds, precision=prec)
        st = [_state(c, gen, 1e-12) for c in clouds]
        for q, c in enumerate(clouds):
            ctx.upload_cloud(q, "Hvoigt", _voigt(c.T, c.freq).cpu().numpy())
        ctx.update_phi_nu(clouds[0].freq.kcore_min, clouds[0].freq.kcore_max)
        s.update(ctx=ctx, params=m1.cloud_params(clouds),
                 state=[_pinned(torch.cat([t[f].reshape(-1) for t in st])) for f in range(3)])
        s["out"] = [m1.pinned_zeros(a.shape) for a in s["state"]]
        return s
    cl, hv, st, gen, rng = _inputs(case, seed)
    s["cloud"] = cl
    s["step"] = dict(c_tilde=cl.c_tilde, dt=cl.dt, z_center=cl.z_center, bc_r_right=cl.bc_r_right,
                     bc_z_bot=cl.bc_z_bot, bc_z_top=cl.bc_z_top)
    s["state"] = [_pinned(t) for t in st]
    if kind == "bands":
        # broad bands: gray opacities per band, all bands advected
        w = torch.rand(hv.shape, generator=gen, device=hv.device, dtype=torch.float64)
        ctx = m1.context_for_cloud(cl, precision=prec, hvoigt=hv.cpu().numpy(), alpha_F=(5.0 * w / K.pc).cpu().numpy())
    else:
        ctx = m1.context_for_cloud(cl, precision=prec, hvoigt=hv.cpu().numpy())
    s["ctx"] = ctx
    if kind == "adjoint":
        s["w_spec"] = rng.uniform(0.0, 1e10, size=cl.n_nu)
    if kind == "rhd":
        sp, rho = W.rhd_gas_state(cl, seed)
        s["gas"] = {k: np.ascontiguousarray(v) for k, v in sp.items()}
        s["rho"] = rho
        s["sub_dt"] = [np.full((cl.nz, cl.nr), 0.2 * cl.dt) * rng.uniform(0.5, 1.0, size=(cl.nz, cl.nr))
                       for _ in range(2)]
    if kind != "host":
        s["out"] = [m1.pinned_zeros(a.shape) for a in s["state"]]
    return s


def _upload(s):
    for name, a in zip(FIELDS, s["state"]):
        s["ctx"].upload(name, a)


def _download(s):
    # M1Context's own method: for a batch, every cloud's values one after another
    return [m1.M1Context.download(s["ctx"], name, out=o) for name, o in zip(FIELDS, s["out"])]


def run(s):
    c, ctx, kind = s["case"], s["ctx"], s["kind"]
    if kind == "host":
        J, Hr, HZ, rec = ctx.static_step_host(*s["state"], out=s["state"], **s["step"])
        return [rec, J, Hr, HZ]
    _upload(s)
    if kind == "run":
        rec = ctx.static_steps(c["steps"], **s["step"])
    elif kind == "batch":
        rec = ctx.batch_steps(c["steps"], s["params"])
    elif kind == "adjoint":
        every = c["every"]
        g = ctx.adjoint(c["steps"], w_MF=1.0, w_spec=s["w_spec"], checkpoint_every=every, **s["step"])
        return [g["M_F"], g["spectrum"], g["grad_alpha"], g["grad_alpha_c"], g["grad_T"], g["grad_Hv"],
                g["grad_u_r_star"], g["grad_u_Z_star"], g["grad_J0"], g["grad_H_r0"], g["grad_H_Z0"]]
    elif kind == "phases":
        p = s["step"]
        ctdt = p["c_tilde"] * p["dt"]
        rec = []
        for _ in range(c["steps"]):
            ctx.advect(ctdt, p["bc_r_right"], p["bc_z_bot"], p["bc_z_top"])
            ctx.emission_absorption(p["c_tilde"], p["dt"])
            ctx.frequency_update(ctdt)
            mf = ctx.force_multiplier(p["dt"], p["z_center"], p["bc_z_bot"])
            rec.append([*mf, ctx.f_esc(mf[3], p["bc_z_bot"])])
            ctx.reset_dru()
        rec = np.array(rec)
    elif kind == "rhd":
        p, sp = s["step"], s["gas"]
        ctdt = p["c_tilde"] * p["dt"]
        ctx.rhd_lya_prepare(sp["T"], sp["nHI"], sp["nH2"], sp["nHII"], sp["nHeI"], sp["ne"], sp["nOHx"], sp["nCHx"],
                            s["rho"], W.DUST_KAPPA_ABS, W.DUST_KAPPA_F, W.DUST_RHO_IGNORE)
        ctx.advect(ctdt, p["bc_r_right"], p["bc_z_bot"], p["bc_z_top"])
        r = [ctx.rhd_lya_absorb(dt, p["c_tilde"], commit=True) for dt in s["sub_dt"]]
        ctx.frequency_update(ctdt)
        rec = [[q["reject"], q["e_new"], q["dru_r"], q["dru_Z"], q["split"]] for q in r]
    else:                                                     # bands
        p = s["step"]
        ctdt = p["c_tilde"] * p["dt"]
        for _ in range(c["steps"]):
            ctx.advect_jh(ctdt, 0, c["nnu"] - 1, False, p["bc_r_right"], p["bc_z_bot"], p["bc_z_top"])
        rec = []
    return [rec, *_download(s)]


# ---- the same in plain torch, 64 bits -----------------------------------------------------------

JEPS, HEPS, FMIN, FMAX, PMIN, PMAX = 1e-60, 1e-100, 1e-10, 1.0 - 1e-10, 1e-3, 40.0


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_device())


def _sqrt(x):
    """sqrt with a zero derivative at 0."""
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))), torch.zeros_like(x))


def _inv(x):
    nz = x != 0
    return torch.where(nz, 1.0 / torch.where(nz, x, torch.ones_like(x)), torch.zeros_like(x))


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _eddington(f, nr, nz, on):
    f = torch.clamp(f, max=FMAX)
    chi = (3.0 + 4.0 * f * f) / (5.0 + 2.0 * torch.sqrt(4.0 - 3.0 * f * f))
    a, b = 0.5 * (1.0 - chi), 0.5 * (3.0 * chi - 1.0)
    third = torch.full_like(f, 1.0 / 3.0)
    return (torch.where(on, a + b * nr * nr, third), torch.where(on, a + b * nz * nz, third),
            torch.where(on, b * nr * nz, torch.zeros_like(f)))


def _closure(J, Hr, HZ):
    H2 = Hr * Hr + HZ * HZ
    on = ~((J <= JEPS) | (H2 <= HEPS * HEPS) | (H2 <= FMIN * FMIN * J * J))
    H = _sqrt(torch.where(on, H2, torch.zeros_like(H2)))
    f = torch.clamp(H / torch.where(on, J, torch.ones_like(J)), min=FMIN)
    iH = _inv(H)
    return _eddington(f, Hr * iH, HZ * iH, on)


def _hll(f, mu):
    f, mu = torch.clamp(f, FMIN, FMAX), torch.clamp(mu, -1.0, 1.0)
    sq = torch.sqrt(4.0 - 3.0 * f * f)
    fac = _sqrt(torch.clamp(2.0 / 3.0 * (4.0 - 3.0 * f * f - sq) + 2.0 * mu * mu * (2.0 - f * f - sq), min=0.0))
    return torch.clamp((mu * f - fac) / sq, -1, 1), torch.clamp((mu * f + fac) / sq, -1, 1)


def _faces(c, aF, iv, uc, zdir, hll):
    """Fluxes of (J, H_r, H_Z) through a set of faces and K_phiphi on their two sides; c: the four
    stencil cells as (J, H_r, H_Z), iv: their intervals, uc: u*/c."""
    q = [(J, Hr / torch.clamp(J, min=JEPS), HZ / torch.clamp(J, min=JEPS)) for J, Hr, HZ in c]
    left, right = [], []
    for n in range(3):
        d = (q[2][n] - q[1][n]) * iv[3]
        left.append(q[1][n] + _minmod((q[1][n] - q[0][n]) * iv[2], d) * iv[0])
        right.append(q[2][n] - _minmod((q[3][n] - q[2][n]) * iv[4], d) * iv[1])
    side = []
    for J, fr, fZ in (left, right):
        J = torch.clamp(J, min=JEPS)
        f = _sqrt(fr * fr + fZ * fZ)
        over = f > 1.0
        i = torch.where(over, _inv(f), torch.ones_like(f))
        fr, fZ, f = fr * i, fZ * i, torch.where(over, torch.ones_like(f), f)
        i = _inv(f)
        nr, nz = fr * i, fZ * i
        Drr, DZZ, DrZ = _eddington(f, nr, nz, f > FMIN)
        kp = torch.clamp(1.0 - Drr - DZZ, 0.0, 1.0) * J
        H = (fr * J, fZ * J)
        F = (H[1], DrZ * J, DZZ * J) if zdir else (H[0], Drr * J, DrZ * J)
        side.append(dict(U=(J, *H), F=F, k=kp, f=f, n=nz if zdir else nr))
    L, R = side
    tau = aF[0] * iv[0] + aF[1] * iv[1]
    eps = (0.2 + tau) / (0.2 + tau + tau * tau)
    diff = -(c[2][0] - c[1][0]) / (3.0 * torch.clamp(tau, min=1e-300))
    out = []
    if hll:
        (l1, l3), (r1, r3) = _hll(L["f"], L["n"]), _hll(R["f"], R["n"])
        SR, SL = torch.clamp(torch.maximum(l3, r3), min=0.0), torch.clamp(torch.minimum(l1, r1), max=0.0)
        for n in range(3):
            h = (SR * L["F"][n] - SL * R["F"][n] + SR * SL * (R["U"][n] - L["U"][n])) / \
                torch.clamp(SR - SL, min=1e-300)
            out.append(eps * h + (1.0 - eps) * (diff if n == 0 else 0.5 * (L["F"][n] + R["F"][n])))
    else:
        for n in range(3):
            m, j = 0.5 * (L["F"][n] + R["F"][n]), 0.5 * (R["U"][n] - L["U"][n])
            out.append(eps * (m - j) + (1.0 - eps) * diff if n == 0 else m - eps * j)
    return [o + uc * torch.where(uc < 0, R["U"][n], L["U"][n]) for n, o in enumerate(out)], L, R


def _ghosts(U, dim, lo, hi):
    """Two ghost cells on either side along `dim` (0: Z, 1: r); 0 reflects, 1 lets flow out."""
    n = U[0].shape[dim]
    comp = 2 if dim == 0 else 1
    out = []
    for f, x in enumerate(U):
        def cell(i):
            return x.narrow(dim, i, 1)
        if lo == 0:
            a = [cell(1), cell(0)]
            a = [-v for v in a] if f == comp else a
        else:
            a = [torch.clamp(cell(0), max=0.0) if f == comp else cell(0)] * 2
        if hi == 0:
            b = [cell(n - 1), cell(n - 2)]
            b = [-v for v in b] if f == comp else b
        else:
            b = [torch.clamp(cell(n - 1), min=0.0) if f == comp else cell(n - 1)] * 2
        out.append(torch.cat([*a, x, *b], dim))
    return out


def _intervals(L, R, a, b, c, bnd):
    n = len(L)
    iv = np.empty((n + 1, 5))
    iv[0], iv[n] = bnd[:5], bnd[5:]
    iv[1:n] = np.stack([L, R, a, b, c], 1)[:n - 1]
    return iv


class _Exact:
    """One static-driver iteration on torch tensors [Z, r, bin], written from the equations."""

    def __init__(self, cl, hv, aF=None):
        g, f = cl.geom, cl.freq
        self.cl, self.core = cl, (f.kcore_min, f.kcore_max)
        self.ri = _t(_intervals(g.dr_L, g.dr_R, g.inv_dr_i_im1, g.inv_dr_ip1_i, g.inv_dr_ip2_ip1, g.dr_b))
        self.zi = _t(_intervals(g.dZ_L, g.dZ_R, g.inv_dZ_j_jm1, g.inv_dZ_jp1_j, g.inv_dZ_jp2_jp1, g.dZ_b))
        for n in ("dV", "inv_dV", "A_r", "A_Z"):
            setattr(self, n, _t(getattr(g, n))[:, :, None])
        self.irc = _t(g.inv_r_cell)[None, :, None]
        for n in ("alpha", "alpha_c", "alpha_cF", "pd", "js", "T", "dur_dr", "dur_dZ", "duZ_dr", "duZ_dZ",
                  "ur_over_r", "u_r_star", "u_Z_star"):
            setattr(self, n, _t(getattr(cl, n))[:, :, None])
        for n in ("nu", "nuC", "dnu", "inv_dnu", "inv_nuC"):
            setattr(self, n, _t(getattr(f, n)))
        self.hv, self.aF0 = hv, aF
        self.hll = cl.flux_method == W.FLUX_HLL

    def flux_opacity(self):
        return self.aF0 if self.aF0 is not None else self.alpha * self.hv + self.alpha_cF

    def window(self, J):
        e = (torch.clamp(J - 10 * JEPS, min=0.0) * self.dnu * self.dV).sum((0, 1))
        tot = (torch.clamp(J - JEPS, min=0.0) * self.dnu * self.dV).sum()
        on = torch.nonzero(e > 1e-10 * tot).flatten()
        lo, hi = (int(on[0]), int(on[-1])) if on.numel() else (J.shape[2] - 1, 0)
        return min(lo, self.core[0]), max(hi, self.core[1])

    def advect(self, J, Hr, HZ, k0, k1):
        cl, ctdt = self.cl, self.cl.c_tilde * self.cl.dt
        s = slice(k0, k1 + 1)
        U = [x[:, :, s] for x in (J, Hr, HZ)]
        aF = self.flux_opacity()[:, :, s]
        nz, nr = U[0].shape[:2]
        P = _ghosts(U, 1, 0, cl.bc_r_right)
        A = torch.cat([aF[:, :1], aF, aF[:, -1:]], 1)
        iv = [self.ri[:, q][None, :, None] for q in range(5)]
        F, L, R = _faces([[p[:, d:d + nr + 1] for p in P] for d in range(4)], (A[:, :-1], A[:, 1:]), iv,
                         self.u_r_star / K.c, False, self.hll)
        # K_phiphi on the axis: only the Z component of the flux is left there
        J0, Z0 = R["U"][0][:, :1], R["U"][2][:, :1]
        fz = torch.clamp(Z0 / J0, -1.0, 1.0)
        D = _eddington(fz.abs(), torch.zeros_like(fz), torch.sign(fz), fz.abs() > FMIN)
        kR = torch.cat([torch.clamp(1.0 - D[0] - D[1], 0.0, 1.0) * J0, R["k"][:, 1:]], 1)
        kav = 0.5 * (L["k"][:, 1:] + kR[:, :-1])
        dU = [self.A_r[:, 1:] * x[:, 1:] - self.A_r[:, :-1] * x[:, :-1] for x in F]
        del F, L, R, P
        P = _ghosts(U, 0, cl.bc_z_bot, cl.bc_z_top)
        A = torch.cat([aF[:1], aF, aF[-1:]], 0)
        iv = [self.zi[:, q][:, None, None] for q in range(5)]
        F, _, _ = _faces([[p[d:d + nz + 1] for p in P] for d in range(4)], (A[:-1], A[1:]), iv, self.u_Z_star / K.c,
                         True, self.hll)
        dU = [d + self.A_Z[1:] * x[1:] - self.A_Z[:-1] * x[:-1] for d, x in zip(dU, F)]
        del F, P
        n = [u - ctdt * self.inv_dV * d for u, d in zip(U, dU)]
        cc = ctdt / K.c
        Jn = torch.clamp(n[0], min=JEPS) - cc * self.work_term(*U) * U[0]
        hr = n[1] + ctdt * kav * self.irc - cc * (U[1] * self.dur_dr + U[2] * self.dur_dZ)
        hz = n[2] - cc * (U[1] * self.duZ_dr + U[2] * self.duZ_dZ)
        new = self.causal(torch.clamp(Jn, min=JEPS), hr, hz)
        return [torch.cat([x[:, :, :k0], y, x[:, :, k1 + 1:]], 2) for x, y in zip((J, Hr, HZ), new)]

    @staticmethod
    def causal(J, hr, hz):
        H2 = hr * hr + hz * hz
        over = H2 > J * J
        f = torch.where(over, J * _inv(_sqrt(torch.where(over, H2, torch.zeros_like(H2)))), torch.ones_like(J))
        return J, hr * f, hz * f

    def work_term(self, J, Hr, HZ):
        Drr, DZZ, DrZ = _closure(J, Hr, HZ)
        return Drr * self.dur_dr + DrZ * (self.dur_dZ + self.duZ_dr) + DZZ * self.duZ_dZ + \
            torch.clamp(1.0 - Drr - DZZ, min=0.0) * self.ur_over_r

    def emission(self, J, Hr, HZ):
        """Returns the new state and the momentum Delta rho u of each cell."""
        ct, dt = self.cl.c_tilde, self.cl.dt
        k0, k1 = self.core
        core = torch.zeros_like(self.dnu)
        core[k0:k1 + 1] = 1.0
        phi = core * self.hv / (core * self.dnu * self.hv).sum(2, keepdim=True)
        Jn = (J + self.js * ct * phi * dt) / (1.0 + (self.alpha_c + self.alpha * self.pd * self.hv) * ct * dt)
        i = 1.0 / (1.0 + self.flux_opacity() * ct * dt)
        hr, hz = Hr * i, HZ * i
        k4 = 4.0 * math.pi / K.c / ct
        return (Jn, hr, hz), k4 * (self.dnu * (Hr - hr)).sum(2), k4 * (self.dnu * (HZ - hz)).sum(2)

    def frequency(self, J, Hr, HZ):
        dw = 1.0 / (self.cl.c_tilde * self.cl.dt)
        floor = torch.clamp(self.alpha, min=self.cl.alpha_floor)
        dD = K.b_prefact * torch.sqrt(self.T) * (K.nu_lya / K.c)
        Kb = 0.5 * floor * dD * dD * self.hv
        rec = (K.h / K.kB) / self.T
        v = (self.work_term(J, Hr, HZ) / K.c)[:, :, 1:-1]
        nC, iC = self.nuC, self.inv_nuC
        dn = (nC[2:] - self.nu[2:-1], self.nu[2:-1] - nC[1:-1], self.nu[1:-2] - nC[:-2])
        r, P = [], []
        for d, lo in zip(dn, (2, 1, 0)):
            s = slice(lo, lo + J.shape[2] - 2)
            k = Kb[:, :, s]
            c = v * nC[s]
            if self.cl.recoil:
                c = c + k * (rec - 2.0 * iC[s])
            r.append(d / k)
            P.append(torch.clamp(c * r[-1], -PMAX, PMAX))

        def fit(P, sgn):
            """e^{sgn P} and (1 - e^{sgn P}) / P, by their series where |P| is small."""
            t = P.abs() < PMIN
            Ps = torch.where(t, torch.ones_like(P), P)
            e = torch.exp(sgn * Ps)
            return torch.where(t, 1.0 + sgn * P + 0.5 * P * P, e), torch.where(t, -sgn - 0.5 * P, (1.0 - e) / Ps)

        oRp, xRp = fit(P[0], 1.0)
        oL, xL = fit(P[1], -1.0)
        oR, xR = fit(P[1], 1.0)
        oLm, xLm = fit(P[2], -1.0)
        up = self.inv_dnu[1:-1] / (xL * r[1] - xRp * r[0])
        dn_ = self.inv_dnu[1:-1] / (xLm * r[2] - xR * r[1])
        a, c = oLm * dn_, oRp * up
        b = -(oL * up + oR * dn_ + dw)
        d = -dw * J[:, :, 1:-1]
        # elimination down the bins and back; the couplings to the first and the last bin are dropped
        n = b.shape[2]
        cp, dp = [], []
        for k in range(n):
            den = b[..., k] - (a[..., k] * cp[-1] if k else 0.0)
            cp.append(c[..., k] / den)
            dp.append((d[..., k] - (a[..., k] * dp[-1] if k else 0.0)) / den)
        x = [dp[-1]]
        for k in range(n - 2, -1, -1):
            x.append(dp[k] - cp[k] * x[-1])
        Jn = torch.cat([J[:, :, :1], torch.stack(x[::-1], 2), J[:, :, -1:]], 2)
        Jn = torch.clamp(Jn, min=JEPS)
        ratio = Jn / torch.clamp(J, min=JEPS)
        return self.causal(Jn, Hr * ratio, HZ * ratio)

    def record(self, Hr, HZ, dr, dz):
        """M_F, its radial net and outward parts, L and f_esc of one iteration."""
        g, cl = self.cl.geom, self.cl
        fr, fz = dr / cl.dt, dz / cl.dt
        dV = self.dV[..., 0]
        r, z = _t(g.rCoM)[None, :], (_t(g.ZCoM) - cl.z_center)[:, None]
        rad = (fr * r + fz * z) / torch.sqrt(r * r + z * z)
        L = 4.0 * math.pi * (dV * self.js[..., 0]).sum()
        k = K.c / L
        refl = cl.bc_z_bot == W.BC_REFLECT
        esc = (self.A_r[:, -1] * torch.clamp(Hr[:, -1], min=0.0) * self.dnu).sum() + \
              (self.A_Z[-1] * torch.clamp(HZ[-1], min=0.0) * self.dnu).sum()
        if not refl:
            esc = esc + (self.A_Z[0] * torch.clamp(-HZ[0], min=0.0) * self.dnu).sum()
        return [k * (dV * _sqrt(fr * fr + fz * fz)).sum(), k * (dV * rad).sum(),
                k * (dV * torch.clamp(rad, min=0.0)).sum(), (2.0 if refl else 1.0) * L, 4.0 * math.pi * esc / L]

    def step(self, J, Hr, HZ, win=None):
        k0, k1 = win or self.window(J.detach())
        U = self.advect(J, Hr, HZ, k0, k1)
        U, dr, dz = self.emission(*U)
        U = self.frequency(*U)
        return U, self.record(U[1], U[2], dr, dz), (k0, k1)

    def run(self, U, steps, with_window=True):
        recs = []
        for _ in range(steps):
            U, rec, w = self.step(*U)
            recs.append([float(v) for v in rec] + ([float(w[0]), float(w[1])] if with_window else []))
        return np.array(recs), U


def exact(case, seed):
    kind = case["kind"]
    if kind == "rhd":
        return None        # the gas opacities come from fits and tables that would be restated here
    if kind == "batch":
        gen, _ = _rng(seed)
        clouds = _batch_clouds(case, seed)
        recs, out = [], [[], [], []]
        for c in clouds:
            U = _state(c, gen, 1e-12)
            e = _Exact(c, _voigt(c.T, c.freq).reshape(U[0].shape))
            rec, U = e.run(U, case["steps"])
            recs.append(rec)
            for o, u in zip(out, U):
                o.append(u.reshape(-1))
        return [np.stack(recs, 1), *[torch.cat(o) for o in out]]
    cl, hv, U, gen, rng = _inputs(case, seed)
    if kind == "bands":
        w = torch.rand(hv.shape, generator=gen, device=hv.device, dtype=torch.float64)
        e = _Exact(cl, hv, 5.0 * w / K.pc)
        for _ in range(case["steps"]):
            U = e.advect(*U, 0, case["nnu"] - 1)
        return [[], *U]
    e = _Exact(cl, hv)
    if kind == "adjoint":
        return _exact_adjoint(case, e, U, rng.uniform(0.0, 1e10, size=cl.n_nu))
    if kind == "host":
        rec, U = e.run(U, 1)
        return [rec[0], *U]
    rec, U = e.run(U, case["steps"], with_window=kind != "phases")
    return [rec, *U]


def _exact_adjoint(case, e, U, w_spec):
    """Reverse mode of torch through the same iterations; every iteration keeps only its input."""
    cl, n = e.cl, case["steps"]
    names = ("alpha", "alpha_c", "T", "hv", "u_r_star", "u_Z_star")
    with torch.no_grad():
        states, wins, S = [], [], U
        for _ in range(n):
            states.append(S)
            S, rec, w = e.step(*S)
            wins.append(w)
    nz, nr = cl.nz, cl.nr
    ring = [(j, nr - 2) for j in range(1, nz - 1)] + [(nz - 2, i) for i in range(1, nr - 2)] + \
        [(1, i) for i in range(1, nr - 2)]
    jj = torch.tensor([q[0] for q in ring], device=U[0].device)
    ii = torch.tensor([q[1] for q in ring], device=U[0].device)
    spec = S[0][jj, ii].mean(0)
    lam = [torch.zeros_like(x) for x in U]
    lam[0].index_put_((jj, ii), _t(w_spec)[None, :].expand(len(ring), -1) / len(ring), accumulate=True)
    keep = {k: getattr(e, k) for k in names}
    grad = {k: torch.zeros_like(v) for k, v in keep.items()}
    for q in range(n - 1, -1, -1):
        x = [u.detach().requires_grad_(True) for u in states[q]]
        p = [keep[k].detach().requires_grad_(True) for k in names]
        for k, v in zip(names, p):
            setattr(e, k, v)
        y, r, _ = e.step(*x, win=wins[q])
        obj = sum((a * b).sum() for a, b in zip(y, lam)) + (r[0] if q == n - 1 else 0.0)
        gr = torch.autograd.grad(obj, x + p, allow_unused=True)
        lam = [v if v is not None else torch.zeros_like(u) for u, v in zip(x, gr[:3])]
        for k, v in zip(names, gr[3:]):
            if v is not None:
                grad[k] += v
        del x, p, y, r, obj, gr
    g = {k: (v if k == "hv" else v[..., 0]) for k, v in grad.items()}
    return [float(rec[0]), spec, g["alpha"], g["alpha_c"], g["T"], g["hv"], g["u_r_star"], g["u_Z_star"], *lam]

"""Workloads of the dycore as its users call it, for timing and for checking results.

Every case goes through the package's public entry points with inputs built on
the GPU from a seed: terrain, a stratified balanced column, sheared wind with
noise, clouds, map factors, and drifting boundary strips.  Kinds:

* ``step``      one RK3 step: ``dycore.rk_scan_step`` (the drop-in call),
                ``dycore.Stepper.step_into`` (the call of a time loop) or a
                captured CUDA graph of it;
* ``forecast``  ``dycore.forecast_step``: the step, the guards and the
                end-of-step lateral boundary pass;
* ``batch``     ``dycore.BatchStepper.step_into`` over ensemble members, in a
                captured CUDA graph;
* ``tower``     ``nesting.NestTower.run``: a parent step, the boundary package,
                three child steps, the two-way feedback;
* ``advect``    ``adjoint.scalar_advection`` and its backward pass;
* ``acoustic``  ``adjoint.acoustic_loop`` and its backward pass.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from wrf_gpu_b200 import _capi, adjoint, dycore, nesting

R_D, CP_D, P0, G, T0 = 287.0, 1004.5, 1.0e5, 9.81, 300.0
F64 = torch.float64
MOIST = dycore.MOIST


def _case(kind, nx, ny, nz, **kw):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, call="into", boundary="specified", moist=1, scalar=0, ns=6, dt=6.0,
             dx=1000.0, hmax=2000.0, stretch=False, lid=False, damp=False, w_damping=False, hyps=1, diff6=False,
             smag=False, precision="fp64", physics=False, members=1, nsub=6)
    c.update(kw)
    return c


def listed():
    return [
        # a small window driven through the drop-in call: launches and host work count
        dict(_case("step", 40, 32, 50, call="scan"), name="window_40x32x50"),
        # the idealised dry warm bubble: doubly periodic, rigid lid
        dict(_case("step", 64, 64, 40, boundary="periodic", moist=0, lid=True, hmax=0.0), name="bubble_64x64x40"),
        # the 9 km nest level, with the physics tendencies of a coupled run
        dict(_case("step", 150, 150, 45, call="scan", physics=True, dx=9000.0, dt=54.0), name="physics_150x150x45"),
        # two ensemble members in one captured call
        dict(_case("batch", 129, 129, 45, members=2), name="members_2x129x129x45"),
        # monotonic limiters on theta and moisture, odd sizes, log-pressure hypsometry
        dict(_case("step", 217, 185, 35, boundary="periodic", moist=2, scalar=2, hyps=2, ns=4), name="monotonic_217x185x35"),
        # mountain wave: dry, stretched levels, Rayleigh layer
        dict(_case("step", 256, 256, 50, moist=0, dx=2000.0, dt=12.0, hmax=1000.0, stretch=True, damp=True),
             name="wave_256x256x50"),
        # an operational forecast step: full boundary pass, 6th-order filter, Smagorinsky, w damping
        dict(_case("forecast", 301, 301, 45, dx=3000.0, dt=18.0, diff6=True, smag=True,
                   w_damping=True, damp=True, call="scan"), name="forecast_301x301x45"),
        # the mixed-precision variant of the step
        dict(_case("step", 301, 301, 50, precision="mixed"), name="mixed_301x301x50"),
        # the headline domain
        dict(_case("step", 433, 433, 50, hmax=3000.0), name="real_433x433x50"),
        # one step of a two-way nest: a parent and its 3:1 child
        dict(_case("tower", 100, 100, 45, boundary="cadence", dx=3000.0, dt=18.0, hmax=300.0, call="scan"),
             name="nest_100x100x45"),
        # gradients of the advection operator for the field and the velocities
        dict(_case("advect", 433, 433, 50, boundary="periodic", moist=0), name="advect_grad_433x433x50"),
        # gradients through an acoustic loop of six small steps
        dict(_case("acoustic", 256, 256, 50, boundary="periodic", moist=0), name="acoustic_grad_256x256x50"),
    ]


def draw(rng):
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["step", "step", "step", "forecast", "batch", "tower", "advect", "acoustic"])
    nz = rng.randint(20, 60)
    if kind == "step":
        boundary = rng.choice(["periodic", "specified", "specified", "cadence", "nested"])
        moist = rng.choice([0, 1, 1, 2])
        precision = rng.choice(["fp64", "fp64", "mixed"])
        return _case("step", size(24, 400), size(24, 400), min(nz, 50), call=rng.choice(["scan", "into", "graph"]),
                     boundary=boundary, moist=moist, scalar=rng.choice([0, 0, 1, 2]), ns=rng.choice([4, 6]),
                     hyps=rng.choice([1, 2]), lid=rng.random() < 0.3, damp=rng.random() < 0.5,
                     w_damping=rng.random() < 0.5, stretch=rng.random() < 0.5, precision=precision,
                     physics=rng.random() < 0.2, hmax=rng.choice([300.0, 1000.0, 3000.0]))
    if kind == "forecast":
        # the filter's monotonic switch is a coin toss where the cadence ties the
        # ring to its neighbour, so the two are not drawn together
        diff6 = rng.random() < 0.6
        return _case("forecast", size(40, 330), size(40, 330), min(nz, 50), boundary="specified" if diff6 else "cadence",
                     dx=3000.0, dt=18.0, diff6=diff6, smag=rng.random() < 0.5, w_damping=True, damp=True, call="scan")
    if kind == "batch":
        return _case("batch", size(33, 200), size(33, 200), min(nz, 50), members=2, moist=rng.choice([0, 1]))
    if kind == "tower":
        return _case("tower", size(40, 110), size(40, 110), min(nz, 50), boundary="cadence", dx=3000.0, dt=18.0,
                     hmax=300.0, call="scan")
    if kind == "advect":
        return _case("advect", size(40, 433), size(40, 433), nz if nz < 51 else 50, boundary="periodic", moist=0)
    return _case("acoustic", size(32, 256), size(32, 256), min(nz, 50), boundary="periodic", moist=0,
                 nsub=rng.choice([2, 3, 4, 6]), lid=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _waves(g, ny, nx, n=8):
    """A smooth periodic field of n random waves, scaled to 0..1."""
    y = torch.arange(ny, dtype=F64, device="cuda")[:, None] / ny
    x = torch.arange(nx, dtype=F64, device="cuda")[None, :] / nx
    k = torch.randint(1, 5, (2, n), generator=g, device="cuda").to(F64)
    ph = torch.rand(n, generator=g, dtype=F64, device="cuda") * 2.0 * math.pi
    h = sum(torch.cos(2.0 * math.pi * (k[0, i] * y + k[1, i] * x) + ph[i]) / (k[0, i] + k[1, i]) for i in range(n))
    h = h.expand(ny, nx)
    return (h - h.min()) / (h.max() - h.min()).clamp_min(1.0e-30)


def _metrics(c, g, p_top):
    """A Lambert-like grid: map factors near 1, Coriolis parameters, rotation angle."""
    ny, nx, nz = c["ny"], c["nx"], c["nz"]
    eta = np.linspace(1.0, 0.0, nz + 1)
    if c["stretch"]:
        eta = 1.0 - (np.exp(2.0 * np.arange(nz + 1) / nz) - 1.0) / (np.exp(2.0) - 1.0)
    dnw = np.diff(eta)
    dn = np.concatenate([dnw[:1], 0.5 * (dnw[1:] + dnw[:-1])])
    fnm, fnp = np.zeros(nz), np.zeros(nz)
    fnp[1:], fnm[1:] = 0.5 * dnw[1:] / dn[1:], 0.5 * dnw[:-1] / dn[1:]
    cof1 = (2.0 * dn[1] + dn[2]) / (dn[1] + dn[2]) * dnw[0] / dn[1]
    cof2 = dn[1] / (dn[1] + dn[2]) * dnw[0] / dn[2]
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device="cuda")
    m = 1.0 + 0.03 * _waves(g, ny, nx)
    mu = torch.cat([m[:, :1], 0.5 * (m[:, 1:] + m[:, :-1]), m[:, -1:]], 1).contiguous()
    mv = torch.cat([m[:1], 0.5 * (m[1:] + m[:-1]), m[-1:]], 0).contiguous()
    ang = 0.1 * (_waves(g, ny, nx) - 0.5)
    lat = 0.7 + 0.1 * _waves(g, ny, nx)
    one, zero = torch.ones_like, torch.zeros_like
    ec = t(0.5 * (eta[1:] + eta[:-1]))
    ef = t(eta)
    return dycore.DycoreMetrics(
        c1h=one(ec), c2h=zero(ec), c3h=ec, c4h=zero(ec), c1f=one(ef), c2f=zero(ef), c3f=ef, c4f=zero(ef),
        dn=t(dn), dnw=t(dnw), rdn=t(1.0 / dn), rdnw=t(1.0 / dnw), fnm=t(fnm), fnp=t(fnp),
        msftx=m.contiguous(), msfty=m.clone(), msfux=mu, msfuy=mu.clone(), msfvx=mv, msfvy=mv.clone(),
        f=1.458e-4 * torch.sin(lat), e=1.458e-4 * torch.cos(lat), sina=torch.sin(ang), cosa=torch.cos(ang),
        cf1=float(fnp[1] + cof1), cf2=float(fnm[1] - cof1 - cof2), cf3=float(cof2), p_top=float(p_top))


def _col(a):
    return a[:, None, None]


def _alpha(theta, p):
    return (R_D / P0) * theta * (p / P0) ** (-(CP_D - R_D) / CP_D)


def _strips(field, g, noise, width=5):
    """Boundary strips (time, side, width, level, side_len) from the edge rows, drifting in time."""
    nl, yl, xl = field.shape
    out = torch.zeros((2, 4, width, nl, max(yl, xl) + 1), dtype=F64, device="cuda")
    for b in range(width):
        out[:, 0, b, :, :yl] = field[:, :, b]
        out[:, 1, b, :, :yl] = field[:, :, xl - 1 - b]
        out[:, 2, b, :, :xl] = field[:, b, :]
        out[:, 3, b, :, :xl] = field[:, yl - 1 - b, :]
    if noise:
        out = out + noise * _randn(g, *out.shape)
    return out


def _state(c, g):
    """Metrics and a balanced, noisy state of the case."""
    ny, nx, nz = c["ny"], c["nx"], c["nz"]
    ztop = 20000.0
    p_top = P0 * (1.0 - G * ztop / (CP_D * T0)) ** (CP_D / R_D)
    m = _metrics(c, g, p_top)
    ht = c["hmax"] * _waves(g, ny, nx)
    mub = P0 * (1.0 - G * ht / (CP_D * T0)) ** (CP_D / R_D) - p_top
    pb = _col(m.c3h) * mub[None] + p_top
    z = CP_D * T0 / G * (1.0 - (pb / P0) ** (R_D / CP_D))
    theta = 295.0 * torch.exp(0.011 ** 2 * z / G) + 0.1 * _randn(g, nz, ny, nx)
    if c["hmax"] == 0.0:  # isentropic, with a warm bubble
        x = (torch.arange(nx, dtype=F64, device="cuda") - 0.5 * nx) * c["dx"]
        y = (torch.arange(ny, dtype=F64, device="cuda") - 0.5 * ny) * c["dx"]
        r = torch.sqrt((x[None, None, :] / 6000.0) ** 2 + (y[None, :, None] / 6000.0) ** 2 + ((z - 4000.0) / 3000.0) ** 2)
        theta = 300.0 + torch.where(r <= 1.0, 2.0 * torch.cos(0.5 * math.pi * r) ** 2, 0.0) + 0.01 * _randn(g, nz, ny, nx)
    alb = _alpha(torch.full_like(theta, T0), pb)
    al = _alpha(theta, pb) - alb
    mass = mub[None].expand(nz, ny, nx)
    phb, php = torch.zeros((2, nz + 1, ny, nx), dtype=F64, device="cuda")
    phb[0] = G * ht
    phb[1:] = phb[:1] + torch.cumsum(-_col(m.dnw) * mass * alb, 0)
    php[1:] = torch.cumsum(-_col(m.dnw) * mass * al, 0)
    alt = -(_col(m.rdnw) * (php[1:] - php[:-1])) / mass + alb
    pp = P0 * ((R_D * theta) / (P0 * alt)) ** (CP_D / (CP_D - R_D)) - pb
    zf = (z / ztop).clamp(0.0, 1.0)
    wind = 5.0 + 15.0 * zf if c["hmax"] else torch.zeros_like(zf)
    u, v = torch.empty((nz, ny, nx + 1), dtype=F64, device="cuda"), torch.empty((nz, ny + 1, nx), dtype=F64, device="cuda")
    u[..., :nx] = wind + 0.5 * _randn(g, nz, ny, nx)
    u[..., nx] = u[..., 0] if c["boundary"] == "periodic" else u[..., nx - 1] + 0.5 * _randn(g, nz, ny)
    v[:, :ny] = 0.3 * wind * (_waves(g, ny, nx) - 0.5) + 0.5 * _randn(g, nz, ny, nx)
    v[:, ny] = v[:, 0] if c["boundary"] == "periodic" else v[:, ny - 1] + 0.5 * _randn(g, nz, nx)
    w = 0.05 * _randn(g, nz + 1, ny, nx)
    w[0] = 0.0
    t = theta * (pb / P0) ** (R_D / CP_D)
    es = 611.2 * torch.exp(17.67 * (t - 273.15) / (t - 29.65))
    qv = 0.8 * 0.622 * es / (pb - es).clamp_min(1.0) * torch.exp(-z / 8000.0)
    cloud = ((z >= 2000.0) & (z <= 6000.0)).to(F64)
    qc = cloud * torch.exp(math.log(1.0e-4) + 0.5 * _randn(g, nz, ny, nx))
    qr = cloud * torch.exp(math.log(5.0e-5) + 0.5 * _randn(g, nz, ny, nx))
    ice = ((z >= 6000.0) & (z <= 11000.0)).to(F64)
    qi = ice * torch.exp(math.log(2.0e-5) + 0.5 * _randn(g, nz, ny, nx))
    qs, qg = 0.5 * qi, 0.2 * qc
    s = dycore.State(u=u, v=v, w=w, theta=theta, p_total=pb + pp, p_perturbation=pp, ph_total=phb + php,
                     ph_perturbation=php, mu_total=mub.clone(), mu_perturbation=torch.zeros_like(mub),
                     qv=qv, qc=qc, qr=qr, qi=qi, qs=qs, qg=qg)
    if c["boundary"] != "periodic":
        side = max(nx, ny) + 1
        fit = lambda a: torch.nn.functional.pad(a, (0, side - a.shape[-1])) if a.shape[-1] < side else a[..., :side].contiguous()
        for name, f, noise in (("u", u, 0.5), ("v", v, 0.5), ("w", w, 0.05), ("theta", theta, 0.3),
                               ("ph", php, 20.0), ("mu", s.mu_perturbation[None], 30.0), ("p", pp, 20.0),
                               ("pb", pb, 0.0), ("mub", mub[None], 0.0), ("phb", phb, 0.0), ("qv", qv, 1.0e-5)):
            setattr(s, name + "_bdy", fit(_strips(f, g, noise)))
        for q in MOIST[1:]:
            setattr(s, q + "_bdy", fit(_strips(getattr(s, q), g, 1.0e-6)))
    return m, s


def _namelist(c, m):
    b = c["boundary"]
    bc = dycore.BoundaryConfig(force_geopotential=b != "nested", nested_ph_relax=b == "nested",
                               nested_w_relax=b == "nested", nested_ph_spec=b == "nested")
    return dycore.OperationalNamelist(
        metrics=m, nx=c["nx"], ny=c["ny"], nz=c["nz"], dx_m=c["dx"], dy_m=c["dx"], dt_s=c["dt"],
        acoustic_substeps=c["ns"], epssm=0.1, hypsometric_opt=c["hyps"], top_lid=c["lid"], run_physics=False,
        run_boundary=b != "periodic", bc_source="ideal" if b == "periodic" else "wrfbdy", boundary_config=bc,
        specified_bdy_cadence=b == "cadence", w_damping=int(c["w_damping"]), damp_opt=3 if c["damp"] else 0,
        dampcoef=0.2 if c["damp"] else 0.0, use_flux_advection=True, scalar_adv_opt=c["scalar"],
        moist_adv_opt=c["moist"], diff_6th_opt=2 if c["diff6"] else 0, diff_opt=1 if c["smag"] else 0,
        km_opt=4 if c["smag"] else 0, precision=c["precision"])


def _physics(s, g, m):
    """Tendencies of the size a physics suite hands over, coupled with the column mass."""
    mu = float(s.mu_total.mean())
    r = lambda t, scale: scale * _randn(g, *t.shape)
    return SimpleNamespace(ru_tendf=r(s.u, 1.0e-4 * mu), rv_tendf=r(s.v, 1.0e-4 * mu), rw_tendf=r(s.w, 1.0e-5 * mu),
                           ph_tendf=None, t_tendf=r(s.theta, 1.0e-4 * mu), mu_tendf=r(s.mu_total, 1.0e-3),
                           h_diabatic=r(s.theta, 1.0e-5), u_save=None, v_save=None, w_save=None, ph_save=None,
                           t_save=None)


def _carry(s):
    return dycore.initial_operational_carry(s)


def _carry_out(c):
    out = {n: getattr(c.state, n) for n in dycore.STATE_FIELDS + MOIST}
    out.update({n: getattr(c, n) for n in dycore.CARRY_FIELDS})
    return out


def _state_out(c):
    out = {n: getattr(c.state, n) for n in dycore.STATE_FIELDS + MOIST}
    out["mudf"] = c.mudf
    return out


def _acoustic_inputs(c, g, m, s):
    """Stage constants and the work state of an acoustic loop, from the state."""
    ny, nx, nz = c["ny"], c["nx"], c["nz"]
    dts = c["dt"] / c["ns"]
    z = lambda *n: torch.zeros(n, dtype=F64, device="cuda")
    mu = s.mu_total
    muu = torch.cat([mu[:, :1], 0.5 * (mu[:, 1:] + mu[:, :-1]), mu[:, -1:]], 1).contiguous()
    muv = torch.cat([mu[:1], 0.5 * (mu[1:] + mu[:-1]), mu[-1:]], 0).contiguous()
    pb = (s.p_total - s.p_perturbation).contiguous()
    alt = _alpha(s.theta, s.p_total)
    c2a = (CP_D / (CP_D - R_D)) * s.p_total / alt
    cqw = z(nz + 1, ny, nx)
    cqw[1:] = 1.0 / (1.0 + 0.005 * torch.rand((nz, ny, nx), generator=g, dtype=F64, device="cuda"))
    # the tridiagonal factors of the implicit w - ph solve
    cof = (0.5 * dts * G * 1.1) ** 2
    a, gamma, alpha = z(nz + 1, ny, nx), z(nz + 1, ny, nx), torch.ones((nz + 1, ny, nx), dtype=F64, device="cuda")
    rdn, rdnw = m.rdn, m.rdnw
    mm = mu * mu
    a[nz] = -2.0 * cof * rdnw[nz - 1] ** 2 * c2a[nz - 1] * (0.0 if c["lid"] else 1.0) / mm
    for k in range(2, nz):
        a[k] = -cqw[k] * cof * rdn[k] * rdnw[k - 1] * c2a[k - 1] / mm
    for k in range(1, nz):
        b = 1.0 + cqw[k] * cof * rdn[k] * (rdnw[k] * c2a[k] + rdnw[k - 1] * c2a[k - 1]) / mm
        cc = -cqw[k] * cof * rdn[k] * rdnw[k] * c2a[k] / mm
        alpha[k] = 1.0 / (b - a[k] * gamma[k - 1])
        gamma[k] = cc * alpha[k]
    b = 1.0 + 2.0 * cof * rdnw[nz - 1] ** 2 * c2a[nz - 1] / mm
    alpha[nz] = 1.0 / (b - a[nz] * gamma[nz - 1])
    mass = float(mu.mean())
    consts = dict(
        u_tend=1.0e-3 * mass * _randn(g, nz, ny, nx + 1), v_tend=1.0e-3 * mass * _randn(g, nz, ny + 1, nx),
        t_tend=1.0e-4 * mass * _randn(g, nz, ny, nx), rw_tend=1.0e-3 * mass * _randn(g, nz + 1, ny, nx),
        ph_tend=1.0e-2 * mass * _randn(g, nz + 1, ny, nx), alt=alt, pb=pb, c2a=c2a,
        cqu=1.0 / (1.0 + 0.005 * torch.rand((nz, ny, nx + 1), generator=g, dtype=F64, device="cuda")),
        cqv=1.0 / (1.0 + 0.005 * torch.rand((nz, ny + 1, nx), generator=g, dtype=F64, device="cuda")), cqw=cqw,
        php=(0.5 * (s.ph_total[1:] + s.ph_total[:-1])).contiguous(), pt1=s.ph_total, a=a, alpha=alpha, gamma=gamma,
        ww_1=10.0 * _randn(g, nz + 1, ny, nx), mut=mu.contiguous(), muu=muu, muv=muv, u_1=s.u, v_1=s.v, w_save=s.w,
        theta=s.theta, phb0=(s.ph_total[0] - s.ph_perturbation[0]).contiguous())
    work = dict(
        u=mass * 0.01 * _randn(g, nz, ny, nx + 1), v=mass * 0.01 * _randn(g, nz, ny + 1, nx),
        w=mass * 0.001 * _randn(g, nz + 1, ny, nx), ph=_randn(g, nz + 1, ny, nx),
        theta_w=mass * 0.01 * _randn(g, nz, ny, nx), t_2ave=0.01 * _randn(g, nz, ny, nx),
        p=_randn(g, nz, ny, nx), pm1=_randn(g, nz, ny, nx), al=1.0e-5 * _randn(g, nz, ny, nx),
        ww=0.1 * _randn(g, nz + 1, ny, nx), mu=0.1 * _randn(g, ny, nx), muts=mu + 0.1 * _randn(g, ny, nx),
        muave=0.1 * _randn(g, ny, nx), mudf=0.01 * _randn(g, ny, nx))
    cot = {n: _randn(g, *t.shape) for n, t in work.items()}
    return consts, work, cot, dts


def _advect_inputs(c, g):
    ny, nx, nz = c["ny"], c["nx"], c["nz"]
    m = _metrics(c, g, 5000.0)
    q = 300.0 + 10.0 * _waves(g, ny, nx)[None] + 0.5 * _randn(g, nz, ny, nx)
    mu = 9.0e4
    ru, rv = mu * (8.0 + 4.0 * _randn(g, nz, ny, nx)), mu * 4.0 * _randn(g, nz, ny, nx)
    rom = 50.0 * _randn(g, nz + 1, ny, nx)
    rom[0], rom[nz] = 0.0, 0.0
    return m, q.contiguous(), ru, rv, rom, _randn(g, nz, ny, nx)


def prepare(case, seed):
    c, g = case, _generator(seed)
    kind = c["kind"]
    if kind == "advect":
        m, q, ru, rv, rom, cot = _advect_inputs(c, g)
        return dict(kind=kind, xs=[t.requires_grad_(True) for t in (q, ru, rv, rom)], cot=cot, nl=_namelist(c, m))
    m, s = _state(c, g)
    nl = _namelist(c, m)
    if kind == "acoustic":
        consts, work, cot, dts = _acoustic_inputs(c, g, m, s)
        return dict(kind=kind, work={n: t.requires_grad_(True) for n, t in work.items()}, cot=cot, nsub=c["nsub"],
                    op=adjoint.AcousticOp(nl, consts, dts))
    if kind == "batch":
        carries, nls = [_carry(s)], [nl]
        for _ in range(1, c["members"]):
            mk, sk = _state(c, g)
            carries.append(_carry(sk))
            nls.append(_namelist(c, mk))
        bs = dycore.BatchStepper(nls)
        outs = bs.alloc_carries(carries)
        return dict(kind="graph", outs=outs, keep=(bs, carries, nls),
                    graph=_capture(lambda: bs.step_into(carries, outs, lead_seconds=c["dt"])))
    if kind == "tower":
        cn = dict(c, nx=c["nx"] // 2 * 3, ny=c["ny"] // 2 * 3, dx=c["dx"] / 3.0, dt=c["dt"] / 3.0, boundary="nested")
        mc, sc = _state(cn, g)
        nlc = _namelist(cn, mc)
        nlc.boundary_config.update_cadence_s = c["dt"]
        grids = {"p": SimpleNamespace(nx=c["nx"], ny=c["ny"]), "c": SimpleNamespace(nx=cn["nx"], ny=cn["ny"])}
        edge = nesting.NestEdge("p", "c", 3, c["nx"] // 5, c["ny"] // 5)
        tower = nesting.NestTower(["p", "c"], [edge], {"p": nl, "c": nlc}, grids, feedback=True)
        return dict(kind=kind, tower=tower, carries={"p": _carry(s), "c": _carry(sc)})
    carry = _carry(s)
    phys = _physics(s, g, m) if c["physics"] else None
    st = dict(kind=kind, call=c["call"], carry=carry, nl=nl, lead=c["dt"], phys=phys)
    if kind == "step" and c["call"] != "scan":
        stp = dycore.Stepper(nl, physics=phys is not None)
        out = stp.alloc_carry(carry)
        st.update(stepper=stp, out=out)
        if c["call"] == "graph":
            st = dict(kind="graph", outs=[out], keep=(stp, carry, phys, nl),
                      graph=_capture(lambda: stp.step_into(carry, out, lead_seconds=c["dt"], physics=phys)))
    return st


def _capture(fn):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fn()
    return graph


def run(st):
    kind = st["kind"]
    if kind == "graph":
        st["graph"].replay()
        return [_carry_out(o) for o in st["outs"]]
    if kind == "step":
        if st["call"] == "scan":
            return _carry_out(dycore.rk_scan_step(st["carry"], st["nl"], lead_seconds=st["lead"],
                                                  physics_tendencies=st["phys"]))
        st["stepper"].step_into(st["carry"], st["out"], lead_seconds=st["lead"], physics=st["phys"])
        return _carry_out(st["out"])
    if kind == "forecast":
        carry, diag = dycore.forecast_step(st["carry"], st["nl"], 1)
        return dict(_carry_out(carry), limited=diag["theta_limited_cell_count"])
    if kind == "tower":
        out = st["tower"].run(st["carries"], 1)
        return {n: _state_out(out[n]) for n in ("p", "c")}
    if kind == "advect":
        tend = adjoint.scalar_advection(*st["xs"], st["nl"])
        return [tend.detach(), *torch.autograd.grad(tend, st["xs"], st["cot"])]
    out = adjoint.acoustic_loop(st["work"], st["op"], st["nsub"])
    names = list(_capi.ACOUSTIC_WORK_FIELDS)
    grads = torch.autograd.grad([out[n] for n in names], [st["work"][n] for n in names], [st["cot"][n] for n in names])
    return {"out": {n: out[n].detach() for n in names}, "grad": dict(zip(names, grads))}


# ---------------------------------------------------------------------------
# Work and tolerance
# ---------------------------------------------------------------------------

def _state_doubles(nx, ny, nz):
    """float64 values of the prognostic state: 10 dry fields and six species."""
    m, u, v, w, s2 = nz * ny * nx, nz * ny * (nx + 1), nz * (ny + 1) * nx, (nz + 1) * ny * nx, ny * nx
    return u + v + w + 3 * m + 2 * w + 2 * s2 + 6 * m


def _carry_doubles(nx, ny, nz):
    m, u, v, w, s2 = nz * ny * nx, nz * ny * (nx + 1), nz * (ny + 1) * nx, (nz + 1) * ny * nx, ny * nx
    return 2 * m + 5 * w + u + v + 4 * s2


def work(case):
    """Inputs read once, outputs written once; operations of the stencils, the
    equation of state and the small steps as the algorithm states them."""
    c = case
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    cells = nx * ny * nz
    kind = c["kind"]
    if kind == "advect":
        return {"bytes": 8.0 * (3 * cells + (nz + 1) * ny * nx) * 2 + 16.0 * cells, "flops": 330.0 * cells}
    if kind == "acoustic":
        work_d = 5 * cells + 3 * (nz + 1) * ny * nx + nz * ny * (nx + 1) + nz * (ny + 1) * nx + 4 * ny * nx
        const_d = 6 * cells + 9 * (nz + 1) * ny * nx + 3 * nz * ny * (nx + 1) + 3 * nz * (ny + 1) * nx
        # forward, recomputed forward and the reverse sweep
        return {"bytes": 8.0 * (4 * work_d + const_d), "flops": 190.0 * 4 * c["nsub"] * cells}

    def step(nx, ny, nz, moist, ns, state_out):
        n = nx * ny * nz
        sub = 1 + max(1, ns // 2) + ns
        d = 2 * _state_doubles(nx, ny, nz) + (0 if state_out else _carry_doubles(nx, ny, nz))
        return 8.0 * d, n * (190.0 * sub + 3 * 520.0 + (6 * (2 * 110.0 + 260.0) if moist else 0.0))

    b, f = step(nx, ny, nz, c["moist"], c["ns"], kind == "tower")
    if kind == "tower":
        bc, fc = step(nx // 2 * 3, ny // 2 * 3, nz, c["moist"], c["ns"], True)
        return {"bytes": b + 3 * bc, "flops": f + 3 * fc}
    return {"bytes": b * c["members"], "flops": f * c["members"]}


def tolerance(case):
    # Four times what contracting every multiply-add of the build changes.  The
    # loosest outputs of a step are differences that nearly cancel (the column
    # mass tendency, p', the work arrays); the mixed variant rounds its face
    # fluxes to 32 bits.
    if case["kind"] == "advect":
        return {"rel": 1.0e-15}
    if case["kind"] == "acoustic":
        return {"rel": 1.0e-13}
    if case["precision"] == "mixed":
        return {"rel": 2.5e-6}
    return {"rel": 1.2e-11}


# ---------------------------------------------------------------------------
# Plain 64-bit results
# ---------------------------------------------------------------------------

def _ref_advect(q, ru, rv, rom, m, dx):
    def h5(vel, a, dim):
        r = lambda n: torch.roll(a, n, dim)
        q_3, q_2, q_1, q0, q1, q2 = r(3), r(2), r(1), a, r(-1), r(-2)
        f6 = (37.0 * (q0 + q_1) - 8.0 * (q1 + q_2) + (q2 + q_3)) / 60.0
        d5 = ((q2 - q_3) - 5.0 * (q1 - q_2) + 10.0 * (q0 - q_1)) / 60.0
        return vel * (f6 - torch.sign(vel) * d5)

    nz = q.shape[0]
    fx, fy = h5(ru, q, -1), h5(rv, q, -2)
    mid = slice(2, nz - 1)
    qm2, qm1, q0, q1 = q[: nz - 3], q[1: nz - 2], q[2: nz - 1], q[3:]
    vel = rom[mid]
    f4 = (7.0 * (q0 + qm1) - (q1 + qm2)) / 12.0
    d3 = ((q1 - qm2) - 3.0 * (q0 - qm1)) / 12.0
    inner = vel * (f4 + torch.sign(-vel) * d3)
    edge = lambda k: (rom[k] * (m.fnm[k] * q[k] + m.fnp[k] * q[k - 1]))[None]
    zero = torch.zeros_like(q[:1])
    fz = torch.cat([zero, edge(1), inner, edge(nz - 1), zero])
    mx = m.msftx[None]
    t = -mx / dx * (torch.roll(fx, -1, -1) - fx) - mx / dx * (torch.roll(fy, -1, -2) - fy)
    return t - _col(m.rdnw) * (fz[1:] - fz[:-1])


def _ref_substep(x, k, m, nl, dts):
    """One acoustic small step on a doubly periodic domain."""
    rdx, rdy = 1.0 / nl.dx_m, 1.0 / nl.dy_m
    nz = x["p"].shape[0]
    xp = lambda f: (torch.cat([f[..., :1], f], -1), torch.cat([f, f[..., -1:]], -1))
    yp = lambda f: (torch.cat([f[..., :1, :], f], -2), torch.cat([f, f[..., -1:, :]], -2))
    mut, muts0 = k["mut"], x["muts"]

    def dpn(ps):
        lo = 0.5 * (m.cf1 * ps[:1] + m.cf2 * ps[1:2] + m.cf3 * ps[2:3])
        mid = 0.5 * (_col(m.fnm[1:]) * ps[1:] + _col(m.fnp[1:]) * ps[:-1])
        hi = 0.5 * (m.cf1 * ps[-1:] + m.cf2 * ps[-2:-1] + m.cf3 * ps[-3:-2]) if nl.top_lid else torch.zeros_like(lo)
        return torch.cat([lo, mid, hi])

    def wind(vel, tend, cq, mass, msf, rms, pair, rd, d):
        pl, pr = pair(x["p"])
        hl, hr = pair(x["ph"])
        al, ar = pair(x["al"])
        tl, tr = pair(k["alt"])
        bl, br = pair(k["pb"])
        gl, gr = pair(k["php"])
        dp = (msf / rms)[None] * 0.5 * rd * mass[None] * (((hr[1:] - hl[1:]) + (hr[:-1] - hl[:-1]))
                                                       + (tl + tr) * (pr - pl) + (al + ar) * (br - bl))
        n = dpn(pl + pr)
        ml, mr = pair(muts0 - mut)
        dp = dp + (msf / rms)[None] * rd * (gr - gl) * (_col(m.rdnw) * (n[1:] - n[:-1]) - 0.5 * (ml + mr)[None])
        dl, dr = pair(x["mudf"])
        return vel + dts * tend - dts * cq * dp + (-0.01 * d * (dr - dl) / rms)[None]

    u = wind(x["u"], k["u_tend"], k["cqu"], k["muu"], m.msfux, m.msfuy, xp, rdx, nl.dx_m)
    v = wind(x["v"], k["v_tend"], k["cqv"], k["muv"], m.msfvy, m.msfvx, yp, rdy, nl.dy_m)
    uc = u + (k["muu"] / m.msfuy)[None] * k["u_1"]
    vc = v + (k["muv"] / m.msfvx)[None] * k["v_1"]
    div = (m.msftx * m.msfty)[None] * (rdy * (vc[:, 1:] - vc[:, :-1]) + rdx * (uc[..., 1:] - uc[..., :-1]))
    dmdt = (_col(m.dnw) * div).sum(0)
    old = muts0 - mut
    new = old + dts * dmdt
    mu = x["mu"] - old + new
    muts = mut + new
    muave = 0.5 * ((1.0 + nl.epssm) * new + (1.0 - nl.epssm) * old)
    inc = _col(m.dnw) * (dmdt[None] + div) / m.msfty[None]
    rows = torch.cat([x["ww"][:1], x["ww"][:1] - torch.cumsum(inc[: nz - 1], 0)]) - k["ww_1"][:nz]
    ww = torch.cat([rows, x["ww"][nz:]])
    th = k["theta"] - T0
    zero = torch.zeros_like(th[:1])
    wdtn = torch.cat([zero, ww[1:nz] * (_col(m.fnm[1:]) * th[1:] + _col(m.fnp[1:]) * th[:-1]), zero])
    e, wst = torch.roll(th, -1, -1), torch.roll(th, 1, -1)
    n, s = torch.roll(th, -1, -2), torch.roll(th, 1, -2)
    flux = 0.5 * rdy * (v[:, 1:] * (n + th) - v[:, :-1] * (th + s)) + 0.5 * rdx * (u[..., 1:] * (e + th) - u[..., :-1] * (th + wst))
    tend = m.msftx[None] * flux + _col(m.rdnw) * (wdtn[1:] - wdtn[:-1])
    thw = x["theta_w"] + m.msfty[None] * dts * k["t_tend"] - dts * m.msfty[None] * tend
    ep, em = 1.0 + nl.epssm, 1.0 - nl.epssm
    t2 = (0.5 * (ep * thw + em * x["t_2ave"]) + muave[None] * T0) / (muts[None] * (T0 + th))
    pt1, w, ph = k["pt1"], x["w"], x["ph"]
    wd = 0.5 * (ww[1:] + ww[:-1]) * _col(m.rdnw) * (pt1[1:] - pt1[:-1])
    r = dts * (k["ph_tend"][1:] + 0.5 * G * em * w[1:])
    r = torch.cat([r[:-1] - dts * (_col(m.fnm[1:]) * wd[1:] + _col(m.fnp[1:]) * wd[:-1]), r[-1:]])
    r = ph[1:] + m.msfty[None] * r / mut[None]
    rhs = torch.cat([zero, r[:-1], torch.zeros_like(r[-1:]) if nl.top_lid else r[-1:]])
    ht = k["phb0"] / G
    hl, hr = xp(ht)
    hs, hn = yp(ht)
    cf = lambda f: m.cf1 * f[0] + m.cf2 * f[1] + m.cf3 * f[2]
    ucf, vcf = cf(k["u_1"]), cf(k["v_1"])
    sx, sy = (hr - hl) * ucf, (hn - hs) * vcf
    w0 = m.msfty * 0.5 * rdy * (sy[1:] + sy[:-1]) + m.msftx * 0.5 * rdx * (sx[:, 1:] + sx[:, :-1])
    c2a, minv = k["c2a"], (1.0 / m.msfty)[None]
    coef = c2a * _col(m.rdnw) / mut[None]
    g2 = ep * (rhs[1:] - rhs[:-1]) + em * (ph[1:] - ph[:-1])
    ta = coef * g2
    buoy = c2a * k["alt"] * t2
    wn = w + dts * k["rw_tend"]
    mid = wn[1:nz] + (minv * k["cqw"][1:nz] * (0.5 * dts * G * _col(m.rdn[1:])) * (ta[1:] - ta[:-1])
                      + dts * G * minv * (_col(m.rdn[1:]) * (buoy[1:] - buoy[:-1]) - muave[None]))
    top = wn[nz] + minv[0] * (-0.5 * dts * G / mut * m.rdnw[-1] ** 2 * 2.0 * c2a[-1] * g2[-1]
                              - dts * G * (2.0 * m.rdnw[-1] * buoy[-1] + muave))
    wn = torch.cat([w0[None], mid, (torch.zeros_like(top) if nl.top_lid else top)[None]])
    f = [wn[0]]
    for i in range(1, nz + 1):
        f.append((wn[i] - k["a"][i] * f[-1]) * k["alpha"][i])
    b = [f[nz]]
    for i in range(nz - 1, 0, -1):
        b.append(f[i] - k["gamma"][i] * b[-1])
    ws = torch.stack([f[0]] + b[::-1])
    phn = torch.cat([ph[:1], rhs[1:] + m.msfty[None] * 0.5 * dts * G * ep * ws[1:] / muts[None]])
    mw = (muts - mut)[None]
    al = -(k["alt"] * mw + _col(m.rdnw) * (phn[1:] - phn[:-1])) / muts[None]
    pp = c2a * (k["alt"] * (thw - mw * th) / (muts[None] * (T0 + th)) - al)
    return dict(u=u, v=v, w=ws, ph=phn, theta_w=thw, t_2ave=t2, p=pp + 0.1 * (pp - x["pm1"]), pm1=pp, al=al, ww=ww,
                mu=mu, muts=muts, muave=muave, mudf=dmdt)


def exact(case, seed):
    """The two differentiable operators in plain torch; a whole step of the
    model has no short plain form and takes minutes in numpy."""
    c, g = case, _generator(seed)
    if c["kind"] == "advect":
        m, q, ru, rv, rom, cot = _advect_inputs(c, g)
        xs = [t.requires_grad_(True) for t in (q, ru, rv, rom)]
        tend = _ref_advect(*xs, m, c["dx"])
        return [tend.detach(), *torch.autograd.grad(tend, xs, cot)]
    if c["kind"] == "acoustic":
        m, s = _state(c, g)
        nl = _namelist(c, m)
        k, work, cot, dts = _acoustic_inputs(c, g, m, s)
        x = {n: t.requires_grad_(True) for n, t in work.items()}
        y = x
        for _ in range(c["nsub"]):
            y = _ref_substep(y, k, m, nl, dts)
        names = list(_capi.ACOUSTIC_WORK_FIELDS)
        grads = torch.autograd.grad([y[n] for n in names], [x[n] for n in names], [cot[n] for n in names],
                                    allow_unused=True)
        grads = [torch.zeros_like(x[n]) if t is None else t for n, t in zip(names, grads)]
        return {"out": {n: y[n].detach() for n in names}, "grad": dict(zip(names, grads))}
    return None

"""The solver's work as timed cases: inputs, one pass through the public entry points, and its value in plain torch.

listed() and draw() name cases as plain dicts, prepare() makes one case's
inputs on the GPU from a seed, run() makes one pass through the calls of
corefl_b200.Context, exact() computes the same outputs with torch in FP64.

The kinds and what they stand for:

air_step            one SSP-RK3 step of air (rk3_step): a 2-D shock tube, replayed as a CUDA graph as small blocks are
                    run, or a periodic curvilinear block with viscous fluxes
air_inviscid        the characteristic WENO5/WENO7 right-hand side of a periodic block with a density front
air_viscous         the second-order viscous right-hand side
air_riemann         Roe or HLLC with first-order, MUSCL or NND2 states
mix_step            one RK3 step of a non-reacting 9-species mixture, mixture-averaged transport included
mix_inviscid        the mixture's WENO right-hand side (2-D tube or 3-D block)
mix_viscous         the mixture's viscous and diffusive right-hand side
reactors            one point-implicit reaction step of a batch of H2/air reactors at all stages of burning
surrogate_forward   the chemistry network's outputs for a table of states
surrogate_gradients loss and gradients of one minibatch
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "corefl-cpc_b200"))

import corefl_b200 as cf  # noqa: E402
import mechanism  # noqa: E402

DEV = "cuda:0"
F64 = torch.float64
R_U, MW_AIR, GAM = 8314.462618, 28.9647, 1.4
R_AIR = R_U / MW_AIR
PR, CFL, EFIX = 0.72, 0.5, 0.125
DT_REACT = 1e-7


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _flow(kind, mx, my, mz, **kw):
    return dict(kind=kind, mx=mx, my=my, mz=mz, **kw)


def listed():
    return [
        # the classic 400 x 7 Sod tube, where launches and latency are all there is
        dict(_flow("air_step", 400, 7, 1, scheme=52), name="sod_step_400x7"),
        # the headline block: curvilinear periodic, WENO7 and viscous fluxes
        dict(_flow("air_step", 257, 257, 257, scheme=72), name="wave_step_257"),
        # one block of a multi-block mesh, ragged in every direction
        dict(_flow("air_inviscid", 161, 113, 97, scheme=72), name="air_weno7_161x113x97"),
        # the same for the viscous right-hand side
        dict(_flow("air_viscous", 145, 130, 99), name="air_viscous_145x130x99"),
        # the robust second-order scheme of start-up runs
        dict(_flow("air_riemann", 193, 101, 89, scheme=2, recon=2), name="air_roe_193x101x89"),
        # a block of a mixing layer, all its stage work
        dict(_flow("mix_step", 97, 49, 33, scheme=72), name="mix_step_97x49x33"),
        # the 2-D reacting shock tube's convective terms at full size
        dict(_flow("mix_inviscid", 2048, 512, 1, scheme=52), name="mix_weno5_2048x512"),
        # diffusion of a mixing-layer block
        dict(_flow("mix_viscous", 128, 65, 63), name="mix_viscous_128x65x63"),
        # a few reactors: the serial substep chain
        dict(kind="reactors", n=1021, name="reactors_1021"),
        # a full batch of reactors
        dict(kind="reactors", n=1048576, name="reactors_1048576"),
        # inference over a table of states
        dict(kind="surrogate_forward", n=1000003, name="surrogate_forward_1000003"),
        # the minibatch of training
        dict(kind="surrogate_gradients", n=8192, name="surrogate_gradients_8192"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng, nodes):
    """Extents of a 3-D block with at most `nodes` nodes, 9 at least each way."""
    while True:
        m = [_log_int(rng, 9, 257) for _ in range(3)]
        if m[0] * m[1] * m[2] <= nodes:
            return m


def draw(rng):
    kind = rng.choice(["air_step", "air_inviscid", "air_viscous", "air_riemann", "mix_step", "mix_inviscid",
                       "mix_viscous", "reactors", "surrogate_forward", "surrogate_gradients"])
    if kind == "air_step" and rng.random() < 0.4:
        return _flow(kind, _log_int(rng, 100, 2048), _log_int(rng, 7, 512), 1, scheme=rng.choice([52, 72]))
    if kind == "mix_inviscid" and rng.random() < 0.4:
        return _flow(kind, _log_int(rng, 64, 2048), _log_int(rng, 7, 512), 1, scheme=rng.choice([52, 72]))
    if kind == "reactors":
        return dict(kind=kind, n=_log_int(rng, 100, 1 << 20))
    if kind == "surrogate_forward":
        return dict(kind=kind, n=_log_int(rng, 1000, 1 << 20))
    if kind == "surrogate_gradients":
        return dict(kind=kind, n=_log_int(rng, 500, 65536))
    m = _block(rng, 400000 if kind.startswith("mix") else 5000000)
    if kind in ("air_viscous", "mix_viscous"):
        return _flow(kind, *m)
    if kind == "air_riemann":
        return _flow(kind, *m, scheme=rng.choice([2, 4]), recon=rng.choice([1, 2, 3]))
    return _flow(kind, *m, scheme=rng.choice([52, 72]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _rand(gen, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(shape, generator=gen, dtype=F64, device=DEV)


def _ngg(case):
    s = case.get("scheme", 72)
    return 4 if s == 72 else 3 if s == 52 else 2


def _grid(case, g, length):
    """Jacobian, metric and unit coordinates on the padded block: a 2-D block is uniform with unit k spacing, a 3-D one
    x = xi + 0.05 sin(2 pi eta) sin(2 pi zeta), continued periodically into the ghosts; central differences."""
    mx, my, mz = case["mx"], case["my"], case["mz"]

    def axis(m):
        return torch.arange(-g - 1, m + g + 1, dtype=F64, device=DEV) / max(m - 1, 1)

    zeta, eta, xi = torch.meshgrid(axis(mz) * (max(mz - 1, 1)) if mz == 1 else axis(mz), axis(my), axis(mx),
                                   indexing="ij")
    if mz == 1:
        x, y, z = xi * length, eta * (length * 0.01 * my), zeta
    else:
        x = (xi + 0.05 * torch.sin(2 * math.pi * eta) * torch.sin(2 * math.pi * zeta)) * length
        y, z = eta * length, zeta * length
    c = slice(1, -1)

    def d(a, ax):
        s, t = [c, c, c], [c, c, c]
        s[ax], t[ax] = slice(2, None), slice(0, -2)
        return 0.5 * (a[tuple(s)] - a[tuple(t)])

    (x1, x2, x3), (y1, y2, y3), (z1, z2, z3) = [(d(a, 2), d(a, 1), d(a, 0)) for a in (x, y, z)]
    jac = (x1 * (y2 * z3 - y3 * z2) + x2 * (y3 * z1 - y1 * z3) + x3 * (y1 * z2 - y2 * z1))
    met = torch.stack([y2 * z3 - y3 * z2, x3 * z2 - x2 * z3, x2 * y3 - x3 * y2,
                       y3 * z1 - y1 * z3, x1 * z3 - x3 * z1, x3 * y1 - x1 * y3,
                       y1 * z2 - y2 * z1, x2 * z1 - x1 * z2, x1 * y2 - x2 * y1]) / jac
    if mz == 1:  # the tube's i ghosts hold the end nodes' values, and so on
        xi, eta, zeta = xi.clamp(0, 1), eta.clamp(0, 1), torch.zeros_like(zeta)
    return jac.contiguous(), met.contiguous(), [a[c, c, c].contiguous() for a in (xi, eta, zeta)]


def _modes(gen, xyz, n=4):
    """A smooth periodic field of zero mean and amplitude about one, from random Fourier modes."""
    out = torch.zeros_like(xyz[0])
    for _ in range(n):
        k = torch.randint(-2, 3, (3,), generator=gen, device=DEV).tolist()
        a, ph = _rand(gen, -0.6, 0.6, 1).item(), _rand(gen, 0, 2 * math.pi, 1).item()
        out += a * torch.sin(2 * math.pi * (k[0] * xyz[0] + k[1] * xyz[1] + k[2] * xyz[2]) + ph)
    return out


def _param(case, viscous, rho_ref, v_ref, ns=0):
    s = case.get("scheme", 72)
    lab, axes = (6, (0, 1)) if case["mz"] == 1 else (8, (0, 1, 2))
    p = dict(dim=2 if case["mz"] == 1 else 3, n_var=5 + ns, n_spec=ns, n_scalar=ns, n_reac=0, inviscid_scheme=s,
             reconstruction=case.get("recon", 2), viscous_order=viscous, entropy_fix_factor=EFIX, Pr=PR, Sc=0.5,
             cfl=CFL, weno_eps_scale=(rho_ref * v_ref) ** 2, v_ref=v_ref, rho_ref=rho_ref, sensor_eps=-1.0)
    return p, [(a, q, lab) for a in axes for q in (-1, 1)]


def _zone(case, g, param, faces, jac, met, bv, sv=None, mech=None):
    mx, my, mz = case["mx"], case["my"], case["mz"]
    P, N, nv = jac.numel(), mx * my * mz, param["n_var"]
    t = dict(jac=jac.reshape(P), metric=met.reshape(9, P), bv=bv.reshape(6, P).contiguous())
    for k, n in (("cv", nv), ("qn", nv), ("mul", 1), ("mach", 1)):
        t[k] = torch.zeros((n, P), dtype=F64, device=DEV)
    t["dq"] = torch.zeros((nv, N), dtype=F64, device=DEV)
    t["dt_local"] = torch.zeros(N, dtype=F64, device=DEV)
    if sv is not None:
        t["sv"] = sv.reshape(-1, P).contiguous()
        for k in ("acoustic_speed", "gamma", "thermal_conductivity", "reaction_timeScale"):
            t[k] = torch.zeros(P, dtype=F64, device=DEV)
        t["rho_D"] = torch.zeros((sv.shape[0], P), dtype=F64, device=DEV)
    ctx = cf.Context(param, faces)
    ctx.bind(mx, my, mz, g, {k: v.data_ptr() for k, v in t.items()})
    if mech is not None:
        ctx.set_mechanism(mech)
    torch.cuda.synchronize()
    return dict(ctx=ctx, t=t)


def _air_state(case, seed):
    """Jacobian, metric and bv of an air case."""
    gen, g, mz = _gen(seed), _ngg(case), case["mz"]
    viscous = case["kind"] in ("air_step", "air_viscous") and mz > 1
    p0 = 1 / GAM
    t0 = p0 / R_AIR
    length = 1.0
    if viscous:  # Re = 1000 of the wave with Sutherland's viscosity at t0
        length = 1000 * 1.7894e-5 * (t0 / 288.16) ** 1.5 * (288.16 + 110) / (t0 + 110)
    jac, met, xyz = _grid(case, g, length)
    bv = torch.zeros((6,) + tuple(jac.shape), dtype=F64, device=DEV)
    if mz == 1:
        right = xyz[0] >= _rand(gen, 0.45, 0.55, 1)
        f = _rand(gen, 0.95, 1.05, 4)
        bv[0] = torch.where(right, 0.125 * f[0], f[1])
        bv[4] = torch.where(right, 0.1 * f[2], f[3])
    elif case["kind"] in ("air_inviscid", "air_riemann"):
        front = torch.sin(2 * math.pi * (xyz[0] + _rand(gen, 0, 1, 1)))
        bv[0] = 1.0 + 0.4 * torch.tanh(front * case["mx"] / 10) + 0.02 * _modes(gen, xyz)
        bv[4] = p0 * (1 + 0.3 * torch.tanh(front * case["mx"] / 10) + 0.02 * _modes(gen, xyz))
        for l, u in ((1, 1.0), (2, 0.2), (3, -0.1)):
            bv[l] = u + 0.1 * _modes(gen, xyz)
    else:
        bv[0] = 1.0 + 0.01 * torch.sin(2 * math.pi * xyz[0]) + 0.005 * _modes(gen, xyz)
        bv[4] = p0 * (1 + 0.005 * _modes(gen, xyz))
        for l, u in ((1, 1.0), (2, 0.0), (3, 0.0)):
            bv[l] = u + 0.02 * _modes(gen, xyz)
    bv[5] = bv[4] / (bv[0] * R_AIR)
    return g, jac, met, bv, _param(case, 2 if viscous else 0, 1.0, 1.0)


def _mixture():
    m = mechanism.load("li2004")
    return m, {s: m.index(s) for s in m.species}


def _mix_state(case, seed):
    """Jacobian, metric, bv and sv of a mixture case: fuel (H2 : N2) and air streams, as a tube or a periodic wave."""
    gen, g, mz = _gen(seed), _ngg(case), case["mz"]
    m, ix = _mixture()
    jac, met, xyz = _grid(case, g, 2e-3)
    yf, ya = torch.zeros(9, dtype=F64, device=DEV), torch.zeros(9, dtype=F64, device=DEV)
    yf[ix["H2"]], yf[ix["N2"]] = 0.0671, 0.9329
    ya[ix["O2"]], ya[ix["N2"]], ya[ix["H2O"]] = 0.2329, 0.7571, 0.01
    if mz == 1:
        zm = torch.where(xyz[0] >= _rand(gen, 0.45, 0.55, 1), 1.0, 0.0).to(F64)
        pres, temp, vel = 101325.0 * (1 + 4 * zm * _rand(gen, 0.9, 1.1, 1)), 600 + 300 * zm, (0.0, 0.0, 0.0)
    else:
        zm = 0.5 + 0.4 * torch.sin(2 * math.pi * xyz[0]) + 0.02 * _modes(gen, xyz)
        pres, vel = 101325.0 * (1 + 0.01 * _modes(gen, xyz)), (50.0, 5.0, -5.0)
        temp = 600 + 50 * torch.sin(2 * math.pi * xyz[1]) + 5 * _modes(gen, xyz)
    shape = (9, 1, 1, 1)
    sv = zm[None] * yf.view(shape) + (1 - zm[None]) * ya.view(shape)
    trace = torch.tensor([1.0 if s in ("H", "O", "OH", "HO2", "H2O2") else 0.0 for s in m.species], dtype=F64, device=DEV)
    sv = sv + 1e-4 * trace.view(shape) * (zm * (1 - zm))[None]
    sv = sv / sv.sum(0)
    mw = torch.tensor(m.mw, dtype=F64, device=DEV).view(shape)
    bv = torch.zeros((6,) + tuple(jac.shape), dtype=F64, device=DEV)
    bv[4], bv[5] = pres, temp
    bv[0] = bv[4] / (R_U * (sv / mw).sum(0) * temp)
    for l in range(3):
        bv[1 + l] = vel[l] + (5.0 * _modes(gen, xyz) if mz > 1 else 0.0)
    viscous = 2 if case["kind"] in ("mix_step", "mix_viscous") else 0
    return g, jac, met, bv, sv, _param(case, viscous, 1.0, 50.0, ns=9)


class _NoReactions:
    """The mechanism's species, thermo and transport without its reactions."""

    def __init__(self, m):
        self._m, self.n_reac = m, 0
        for k in ("reac_type", "rev_type", "order", "A", "b", "Ea", "A2", "b2", "Ea2", "troe_alpha", "troe_t3",
                  "troe_t1", "troe_t2"):
            setattr(self, k, np.zeros(0))
        for k in ("stoi_f", "stoi_b", "third_body_coeff"):
            setattr(self, k, np.zeros((0, 9)))

    def __getattr__(self, k):
        return getattr(self._m, k)


def _reactor_state(case, seed):
    """Constant-volume H2/air reactors, T 1000-1600 K, 1-10 atm, equivalence ratio 0.5-2, from unburnt to burnt, with
    time scales that ask for 4 to 64 substeps of the step."""
    n, gen = case["n"], _gen(seed)
    m, ix = _mixture()
    t0, phi = _rand(gen, 1000, 1600, n), _rand(gen, 0.5, 2.0, n)
    p = 101325.0 * torch.exp(_rand(gen, 0, math.log(10), n))
    c = _rand(gen, 0, 1, n) ** 2
    burn = c * torch.minimum(phi, torch.ones_like(phi))
    x = torch.zeros((9, n), dtype=F64, device=DEV)
    x[ix["H2"]], x[ix["O2"]], x[ix["N2"]], x[ix["H2O"]] = 2 * phi - 1.96 * burn, 1 - 0.98 * burn, 3.76, 1.96 * burn
    for s, a in (("H", 2e-2), ("O", 5e-3), ("OH", 2e-2), ("HO2", 1e-4), ("H2O2", 1e-5)):
        x[ix[s]] = a * c * _rand(gen, 0.5, 1.5, n)
    mw = torch.tensor(m.mw, dtype=F64, device=DEV)[:, None]
    y = x * mw / (x * mw).sum(0)
    temp = t0 + 1500 * c
    rho = p / (R_U * (y / mw).sum(0) * temp)
    gas = _Gas(m)
    h, _ = gas.enthalpy_cp(temp)
    cv = torch.cat([torch.stack([rho, 0 * rho, 0 * rho, 0 * rho, rho * (h * y).sum(0) - p]), rho * y])
    bv = torch.stack([rho, 0 * rho, 0 * rho, 0 * rho, p, temp])
    ts = DT_REACT / (torch.exp(_rand(gen, math.log(4), math.log(64), n)).floor() + 0.5)
    return m, dict(cv=cv, bv=bv, sv=y, reaction_timeScale=ts)


def _surrogate_inputs(case, seed):
    """Raw features (T, ln p, Box-Cox mass fractions, ln dt), targets, weights and the standardisation."""
    n, gen = case["n"], _gen(seed)
    x = torch.empty((n, 12), dtype=F64, device=DEV)
    x[:, 0], x[:, 1], x[:, 11] = _rand(gen, 1000, 3200, n), _rand(gen, 11.5, 13.8, n), math.log(DT_REACT)
    x[:, 2:11] = ((10 ** _rand(gen, -12, 0, n, 9) + 1e-20) ** 0.1 - 1) / 0.1
    x[:, 11] += _rand(gen, -0.2, 0.2, n)
    mean, std = x.mean(0), x.std(0)
    gt = torch.randn((n, 11), generator=gen, dtype=F64, device=DEV)
    gt = torch.sinh(1.5 * gt + 0.4 * ((x[:, :11] - mean[:11]) / std[:11])) * 1e-3
    gt[:, 9] *= 1e3
    gt[:, 10] = -18 + 2 * (x[:, 0] - mean[0]) / std[0]
    scale = gt.abs().median(0).values
    scale[10] = 0
    z = torch.where(scale > 0, torch.asinh(gt / torch.where(scale > 0, scale, 1.0)), gt)
    lo, hi = ((x - mean) / std).min(0).values, ((x - mean) / std).max(0).values
    norm = torch.cat([mean, 1 / std, z.mean(0), z.std(0), lo, hi, scale]).to(torch.float32)
    w = []
    for rows, cols, fi, fo in ((128, 16, 12, 128), (128, 144, 128, 128), (128, 144, 128, 128), (16, 144, 128, 11)):
        a = torch.zeros((rows, cols), dtype=F64, device=DEV)
        lim = math.sqrt(6 / (fi + fo))
        a[:fo, :fi] = _rand(gen, -lim, lim, fo, fi)
        a[:fo, 15 if cols == 16 else 128] = _rand(gen, -0.1, 0.1, fo)
        w.append(a.reshape(-1))
    return x.to(torch.float32), gt.to(torch.float32), torch.cat(w).to(torch.float32), norm


def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("surrogate"):
        x, gt, w, norm = _surrogate_inputs(case, seed)
        m, _ = _mixture()
        ctx = cf.Context(dict(dim=2, n_var=14, n_spec=9, n_scalar=9, n_reac=m.n_reac, chem_advance_method=1), [])
        ctx.surrogate_init(1, m.element_mass_fractions())
        ctx.surrogate_set_params(weights=w.cpu().numpy(), norm=norm.cpu().numpy())
        st = dict(kind=kind, ctx=ctx, x=x, g=gt, n=case["n"])
        if kind == "surrogate_forward":
            st["y"] = torch.zeros((case["n"], 16), dtype=torch.float32, device=DEV)
        else:
            st["grad"] = torch.zeros(cf.SG_NPARAM, dtype=torch.float32, device=DEV)
        return st
    if kind == "reactors":
        m, s = _reactor_state(case, seed)
        n = case["n"]
        ctx = cf.Context(dict(dim=2, n_var=14, n_spec=9, n_scalar=9, n_reac=m.n_reac, chem_advance_method=1, cfl=CFL), [])
        t = {k: v.clone().contiguous() for k, v in s.items()}
        t["jac"] = torch.ones(n, dtype=F64, device=DEV)
        ctx.bind(n, 1, 1, 0, {k: v.data_ptr() for k, v in t.items()})
        ctx.set_mechanism(m)
        return dict(kind=kind, ctx=ctx, t=t, start={k: v.contiguous() for k, v in s.items()})
    if kind.startswith("air"):
        g, jac, met, bv, (param, faces) = _air_state(case, seed)
        st = _zone(case, g, param, faces, jac, met, bv)
    else:
        g, jac, met, bv, sv, (param, faces) = _mix_state(case, seed)
        st = _zone(case, g, param, faces, jac, met, bv, sv, _NoReactions(_mixture()[0]))
    st.update(kind=kind, graph=case["mz"] == 1)
    st["ctx"].properties()
    st["ctx"].cv_from_bv()
    st["ctx"].sync()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "surrogate_forward":
        ctx.surrogate_forward(st["x"].data_ptr(), st["n"], st["y"].data_ptr())
        return st["y"]
    if kind == "surrogate_gradients":
        loss = ctx.surrogate_gradients(st["x"].data_ptr(), st["g"].data_ptr(), st["n"], st["grad"].data_ptr())
        return {"loss": loss, "grad": st["grad"]}
    t = st["t"]
    if kind == "reactors":  # the batch starts from its given state on every pass
        for k, v in st["start"].items():
            t[k].copy_(v)
        ctx.wu_reaction_step(DT_REACT, schedule=1)
        return {k: t[k] for k in ("cv", "bv", "sv", "reaction_timeScale")}
    if kind in ("air_step", "mix_step"):
        ctx.rk3_step(graph=st["graph"], want_dt=False)
        return {k: t[k] for k in ("cv", "bv", "sv", "mul") if k in t}
    t["dq"].zero_()
    if kind in ("air_viscous", "mix_viscous"):
        ctx.viscous()
    else:
        ctx.inviscid()
    return t["dq"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_FACE = {52: 1250, 72: 1900, 2: 300, 4: 200}  # operations of one face of a scheme in air


def work(case):
    kind = case["kind"]
    if kind == "surrogate_forward":
        return {"bytes": case["n"] * (12 + 16) * 4, "flops": case["n"] * 2 * 41216}
    if kind == "surrogate_gradients":
        return {"bytes": case["n"] * (12 + 11) * 4 + 41216 * 8, "flops": case["n"] * 6 * 41216}
    if kind == "reactors":  # about 22 substeps of 10 thousand operations each
        return {"bytes": case["n"] * 8 * 2 * 30, "flops": case["n"] * 22 * 1e4}
    n, nd = case["mx"] * case["my"] * case["mz"], 3 if case["mz"] > 1 else 2
    mix = kind.startswith("mix")
    face = _FACE.get(case.get("scheme"), 0) * (2.6 if mix else 1)
    if kind == "air_step":  # three stages: state, metric, Jacobian, viscosity in, state out; the fluxes' operations
        return {"bytes": n * 8 * 3 * (11 + 11 + 11), "flops": n * 3 * nd * (face + (170 if nd == 3 else 0))}
    if kind == "mix_step":
        return {"bytes": n * 8 * 3 * (29 + 10 + 13 + 41), "flops": n * 3 * (nd * (face + 700) + 3500)}
    if kind == "air_viscous":
        return {"bytes": n * 8 * (4 + 1 + 10 + 4), "flops": n * nd * 170}
    if kind == "mix_viscous":
        return {"bytes": n * 8 * (4 + 9 + 11 + 10 + 13), "flops": n * nd * 700}
    nv = 14 if mix else 5
    return {"bytes": n * 8 * (nv + 2 + 3 * nd + 1 + nv), "flops": n * nd * face}


def tolerance(case):
    kind = case["kind"]
    if kind == "surrogate_forward":
        return {"rel": 1e-2, "max": 0.2}  # BF16 operands, hardware tanh
    if kind == "surrogate_gradients":
        return {"rel": 2e-2, "max": 0.5}
    # FP64.  Against exact() the steps and the reactors are within 2e-15 of the largest values; the right-hand sides,
    # differences of face fluxes, within 5e-13 on the finest grids, where more digits cancel.  A node whose temperature
    # iteration stops one step earlier moves by 1e-11 of its temperature; the largest differences are next to zero.
    return {"rel": 1e-11, "max": 1e-9}


# ---------------------------------------------------------------------------
# the same in plain torch, FP64
# ---------------------------------------------------------------------------
class _Gas:
    """NASA-7 thermodynamics and mixture-averaged transport of a mechanism's species; arrays are (species, ...)."""

    def __init__(self, m):
        def t(a):
            return torch.tensor(np.asarray(a, dtype=np.float64), dtype=F64, device=DEV)

        self.m, self.mw, self.R = m, t(m.mw), R_U / t(m.mw)
        self.t = {k: t(getattr(m, k)) for k in ("t_low", "t_mid", "t_high", "low", "high", "LJ_potent_inv", "vis_coeff",
                                                "ZRotF298", "WjDivWi_to_One4th", "sqrt_WiDivWjPl1Mul8",
                                                "binary_diffusivity_coeff", "kb_over_eps_jk")}

    def col(self, a, T):
        return a.view((-1,) + (1,) * T.dim())

    def coeff(self, T):
        lo = (T[None] < self.col(self.t["t_mid"], T))
        return [torch.where(lo, self.col(self.t["low"][:, j], T), self.col(self.t["high"][:, j], T)) for j in range(7)]

    def enthalpy_cp(self, T):
        a = self.coeff(T)
        tc = torch.minimum(torch.maximum(T[None], self.col(self.t["t_low"], T)), self.col(self.t["t_high"], T))
        cp = a[0] + tc * (a[1] + tc * (a[2] + tc * (a[3] + tc * a[4])))
        h = tc * (a[0] + tc * (a[1] / 2 + tc * (a[2] / 3 + tc * (a[3] / 4 + tc * a[4] / 5)))) + a[5] + cp * (T[None] - tc)
        R = self.col(self.R, T)
        return h * R, cp * R

    def gibbs(self, T):
        a, tc = self.coeff(T), T[None]
        return a[0] * (1 - torch.log(tc)) - tc * (a[1] / 2 + tc * (a[2] / 6 + tc * (a[3] / 12 + tc * a[4] / 20))) + a[5] / tc - a[6]

    def temperature(self, Y, e, T):
        """Newton's iteration on the internal energy, stopped node by node where the step is below 1e-5."""
        R = (Y * self.col(self.R, T)).sum(0)
        T, live = T.clone(), torch.ones_like(T, dtype=torch.bool)
        for _ in range(50):
            h, cp = self.enthalpy_cp(T)
            t1 = T - ((h * Y).sum(0) - R * T - e) / ((cp * Y).sum(0) - R)
            err = (1 - t1 / T).abs()
            T = torch.where(live, t1, T)
            live = live & (err > 1e-5)
            if not bool(live.any()):
                break
        return T, R

    def properties(self, Y, T):
        """gamma, sound speed, viscosity, conductivity, rho D_k."""
        _, cp = self.enthalpy_cp(T)
        c, k = self.col, self.t
        mwc = c(self.mw, T)
        imw, cpm = (Y / mwc).sum(0), (Y * cp).sum(0)
        R = R_U * imw
        gam = cpm / (cpm - R)
        a = torch.sqrt(gam * R * T)
        X = Y / mwc / imw

        def omega(tr):
            return 1.0548 * tr ** -0.15504 + (tr + 0.55909) ** -2.1705

        td = T[None] * c(k["LJ_potent_inv"], T)
        vis = c(k["vis_coeff"], T) * torch.sqrt(T) / (1.147 * td ** -0.145 + (td + 0.5) ** -2)
        t15 = T * torch.sqrt(T)
        mu, lam = torch.zeros_like(T), torch.zeros_like(T)
        for i in range(9):
            Ri, vi, geom = self.R[i], vis[i], int(self.m.geometry[i])
            li = 3.75 * vi * Ri
            if geom:
                tr = T * k["kb_over_eps_jk"][i, i]
                FT = 1 + 0.5 * math.pi ** 1.5 * tr ** -0.5 + (2 + 0.25 * math.pi ** 2) / tr + math.pi ** 1.5 * tr ** -1.5
                rd = k["binary_diffusivity_coeff"][i, i] * t15 / (omega(tr) * Ri * T)
                crot = 10.0 / 3 if geom == 1 else 5.0
                ab = (2.5 * vi - rd) / (math.pi * k["ZRotF298"][i] / FT * vi + crot * vi + 2 * rd)
                dof = 1.0 if geom == 1 else 1.5
                li = li - 5 * dof * ab * vi * Ri + rd * cp[i] + rd * (2 * dof * ab - 2.5) * Ri
            part = torch.zeros_like(T)
            for j in range(9):
                if i == j:
                    part = part + X[j]
                else:
                    num = 1 + torch.sqrt(vi / vis[j]) * k["WjDivWi_to_One4th"][i, j]
                    part = part + num * num * k["sqrt_WiDivWjPl1Mul8"][i, j] * X[j]
            mu = mu + vi * X[i] / part
            lam = lam + li * X[i] / (1.065 * part - 0.065 * X[i])
        eps = 1e-12
        w = (X + eps) * mwc
        den = torch.zeros_like(Y)
        for i in range(9):
            for j in range(i + 1, 9):
                o = omega(T * k["kb_over_eps_jk"][i, j]) / (k["binary_diffusivity_coeff"][i, j] * t15)
                den[i] += (X[j] + eps) * o
                den[j] += (X[i] + eps) * o
        return gam, a, mu, lam, (w.sum(0) - w) / (T * R_U) / den


def _cut(a, g, rng, sh=(0, 0, 0)):
    """a over the node ranges rng ((i0, i1), (j0, j1), (k0, k1)), shifted by sh."""
    s = [slice(g + r[0] + d, g + r[1] + d) for r, d in zip(rng, sh)]
    return a[..., s[2], s[1], s[0]]


def _slabs(m, d, most):
    """The block's node ranges in slabs of at most `most` nodes, the faces' range along d."""
    full = [[0, n] for n in m]
    full[d] = [-1, m[d]]
    ax = 1 if d == 2 else 2
    rows = max(1, int(most // max(1, m[0] * m[1] * m[2] // m[ax])))
    for lo in range(0, m[ax], rows):
        r = [list(x) for x in full]
        r[ax] = [lo, min(m[ax], lo + rows)]
        yield r


def _to_dq(dq, F, r, d, sign):
    dim = 2 - d
    n = next(iter(F.values())).shape[dim]
    s = [slice(x[0], x[1]) for x in r]
    s[d] = slice(0, n - 1)
    for v, f in F.items():
        dq[v][s[2], s[1], s[0]] += sign * (f.narrow(dim, 1, n - 1) - f.narrow(dim, 0, n - 1))


def _weno7(u, eps):
    a = [(-2 * u[0] + 9 * u[1] - 18 * u[2] + 11 * u[3]) / 6, (u[1] - 6 * u[2] + 3 * u[3] + 2 * u[4]) / 6,
         (-2 * u[2] - 3 * u[3] + 6 * u[4] - u[5]) / 6, (-11 * u[3] + 18 * u[4] - 9 * u[5] + 2 * u[6]) / 6]
    b = [-u[0] + 4 * u[1] - 5 * u[2] + 2 * u[3], u[2] - 2 * u[3] + u[4], u[2] - 2 * u[3] + u[4],
         2 * u[3] - 5 * u[4] + 4 * u[5] - u[6]]
    c = [u[q + 3] - 3 * u[q + 2] + 3 * u[q + 1] - u[q] for q in range(4)]
    beta = [s * s + 13 / 12 * t * t + 1043 / 960 * w * w + s * w / 12 for s, t, w in zip(a, b, c)]
    tau = (beta[0] + 3 * beta[1] - 3 * beta[2] - beta[3]) ** 2
    w = [k * (1 + tau / (eps + x) ** 2) for k, x in zip((1 / 35, 12 / 35, 18 / 35, 4 / 35), beta)]
    v = [-3 * u[0] + 13 * u[1] - 23 * u[2] + 25 * u[3], u[1] - 5 * u[2] + 13 * u[3] + 3 * u[4],
         -u[2] + 7 * u[3] + 7 * u[4] - u[5], 3 * u[3] + 13 * u[4] - 5 * u[5] + u[6]]
    return sum(x * y for x, y in zip(w, v)) / sum(w) / 12


def _weno5(u, eps):
    v = [(2 * u[2] + 5 * u[3] - u[4]) / 6, (-u[1] + 5 * u[2] + 2 * u[3]) / 6, (2 * u[0] - 7 * u[1] + 11 * u[2]) / 6]
    beta = [13 / 12 * (u[2] + u[4] - 2 * u[3]) ** 2 + 0.25 * (3 * u[2] - 4 * u[3] + u[4]) ** 2,
            13 / 12 * (u[1] + u[3] - 2 * u[2]) ** 2 + 0.25 * (u[1] - u[3]) ** 2,
            13 / 12 * (u[0] + u[2] - 2 * u[1]) ** 2 + 0.25 * (u[0] - 4 * u[1] + 3 * u[2]) ** 2]
    low = eps + torch.minimum(torch.minimum(beta[0], beta[1]), beta[2])
    w = [k * (low / (eps + x)) ** 2 for k, x in zip((0.3, 0.6, 0.1), beta)]
    return sum(x * y for x, y in zip(w, v)) / sum(w)


def _exact_weno(dq, m, g, scheme, eps, jac, met, cv, bv, gas=None, sound=None):
    """dq -= differences of the characteristic WENO face fluxes (local Lax-Friedrichs splitting, Roe averages, the
    face normal averaged with the node at i + 1)."""
    R = 3 if scheme == 72 else 2
    weno = _weno7 if scheme == 72 else _weno5
    ns = cv.shape[0] - 5
    for d in range(3 if m[2] > 1 else 2):
        for r in _slabs(m, d, 2e6 if ns == 0 else 5e5):
            def pt(a, off):
                sh = [0, 0, 0]
                sh[d] = off
                return _cut(a, g, r, sh)

            P = []
            for off in range(-R, R + 2):
                Q = pt(cv, off)
                k, p, J = pt(met[3 * d:3 * d + 3], off), pt(bv[4], off), pt(jac, off)
                c = pt(sound, off) if gas else torch.sqrt(GAM * R_AIR * pt(bv[5], off))
                U = (Q[1] * k[0] + Q[2] * k[1] + Q[3] * k[2]) / Q[0]
                G = [Q[0] * U] + [Q[1 + l] * U + p * k[l] for l in range(3)] + [(Q[4] + p) * U]
                lam = U.abs() + torch.sqrt((k * k).sum(0)) * c
                P.append((Q, G + [Q[5 + l] * U for l in range(ns)], p, J, lam))
            k = 0.5 * (_cut(met[3 * d:3 * d + 3], g, r) + _cut(met[3 * d:3 * d + 3], g, r, (1, 0, 0)))
            (ql, pl), (qr, pr) = [(P[R + s][0], P[R + s][2]) for s in (0, 1)]
            root = torch.sqrt(ql[0] * qr[0])
            wl, wr = 1 / (ql[0] + root), 1 / (qr[0] + root)
            u = [wl * ql[1 + l] + wr * qr[1 + l] for l in range(3)]
            pr_ = wl * pl + wr * pr
            H = wl * (ql[4] + pl) + wr * (qr[4] + pr)
            if gas:
                Y = wl * ql[5:] + wr * qr[5:]
                rg = (Y * gas.col(gas.R, root)).sum(0)
                T = pr_ / rg
                h, cp = gas.enthalpy_cp(T)
                cpm = (Y * cp).sum(0)
                gam = cpm / (cpm - rg)
                c = torch.sqrt(gam * rg * T)
                beta = (gam * gas.col(gas.R, root) * T - (gam - 1) * h) / (c * c)
            else:
                gam, c = GAM, torch.sqrt(GAM * pr_)
            gm1 = gam - 1
            n = k / torch.sqrt((k * k).sum(0))
            zero = torch.zeros_like(n[0])
            first = n[0].abs() > 0.8
            b1 = torch.stack([torch.where(first, -n[2], zero), torch.where(first, zero, n[2]),
                              torch.where(first, n[0], -n[1])])
            b1 = b1 / torch.sqrt((b1 * b1).sum(0))
            b2 = torch.linalg.cross(n, b1, dim=0)
            b2 = b2 / torch.sqrt((b2 * b2).sum(0))
            U, V, W = [b[0] * u[0] + b[1] * u[1] + b[2] * u[2] for b in (n, b1, b2)]
            al, ic2 = 0.5 * gm1 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2), 1 / (c * c)
            lam = P[0][4]
            for q in P[1:]:
                lam = torch.maximum(lam, q[4])

            def field(L, lb=None, species=None):
                vp, vm = [], []
                for Q, G, _, J, _ in P:
                    if species is None:
                        f, q = [sum(L[j] * A[j] for j in range(5)) for A in (G, Q)]
                        if lb is not None:
                            f = f + lb * sum(beta[j] * G[5 + j] for j in range(ns))
                            q = q + lb * sum(beta[j] * Q[5 + j] for j in range(ns))
                    else:
                        f, q = [A[5 + species] - Y[species] * A[0] for A in (G, Q)]
                    vp.append(0.5 * J * (f + lam * q))
                    vm.append(0.5 * J * (f - lam * q))
                return weno(vp[:-1], eps) + weno(vm[:0:-1], eps)

            acou = [0.5 if gas else None] * 2 + [-1.0 if gas else None]
            c0 = field([0.5 * ic2 * (al + U * c)] + [-0.5 * ic2 * (gm1 * u[l] + n[l] * c) for l in range(3)] + [0.5 * gm1 * ic2], acou[0])
            c4 = field([0.5 * ic2 * (al - U * c)] + [-0.5 * ic2 * (gm1 * u[l] - n[l] * c) for l in range(3)] + [0.5 * gm1 * ic2], acou[1])
            c3 = field([1 - al * ic2] + [gm1 * u[l] * ic2 for l in range(3)] + [-gm1 * ic2], acou[2])
            c1 = field([-V, b1[0], b1[1], b1[2], zero])
            c2 = field([-W, b2[0], b2[1], b2[2], zero])
            s, t = c0 + c3 + c4, c0 - c4
            F = {0: s, 4: H * s - U * c * t + V * c1 + W * c2 - c * c / gm1 * c3}
            for l in range(3):
                F[1 + l] = u[l] * s - n[l] * c * t + b1[l] * c1 + b2[l] * c2
            for j in range(ns):
                cs = field(None, species=j)
                F[5 + j] = Y[j] * s + cs
                F[4] = F[4] - beta[j] * cs * c * c / gm1
            _to_dq(dq, F, r, d, -1.0)


def _exact_viscous(dq, m, g, jac, met, bv, mul, gas=None, sv=None, cond=None, rho_d=None):
    """dq += differences of the second-order viscous face fluxes."""
    nd = 3 if m[2] > 1 else 2
    for d in range(nd):
        for r in _slabs(m, d, 2e6):
            def sh(ax, s, dn=0):
                o = [0, 0, 0]
                o[ax] += s
                o[d] += dn
                return o

            def ave(a):
                return 0.5 * (_cut(a, g, r) + _cut(a, g, r, sh(d, 1)))

            def grad(a, gm):
                dd = [None] * 3
                for ax in range(3):
                    if ax == d:
                        dd[ax] = _cut(a, g, r, sh(d, 1)) - _cut(a, g, r)
                    else:
                        dd[ax] = 0.25 * (_cut(a, g, r, sh(ax, 1)) - _cut(a, g, r, sh(ax, -1)) +
                                         _cut(a, g, r, sh(ax, 1, 1)) - _cut(a, g, r, sh(ax, -1, 1)))
                return [dd[0] * gm[l] + dd[1] * gm[3 + l] + dd[2] * gm[6 + l] for l in range(3)]

            gm = ave(met)
            gk = ave(met[3 * d:3 * d + 3] * jac)
            mu = ave(mul)
            du = [grad(bv[1 + l], gm) for l in range(3)]
            div = du[0][0] + du[1][1] + du[2][2]
            F = {}
            for a in range(3):
                F[1 + a] = sum(gk[b] * mu * (du[a][b] + du[b][a] - (2.0 / 3 * div if a == b else 0)) for b in range(3))
            dT = grad(bv[5], gm)
            lam = ave(cond) if gas else mu * (GAM * R_AIR / (GAM - 1) / PR)
            F[4] = sum(ave(bv[1 + l]) * F[1 + l] + lam * gk[l] * dT[l] for l in range(3))
            if gas:
                yk, D, imw = ave(sv), ave(rho_d), 1 / gas.mw
                gy = torch.stack([sum(gk[l] * y for l, y in enumerate(grad(sv[j], gm))) for j in range(9)])
                col = (9, 1, 1, 1)
                gw = (gy * imw.view(col)).sum(0) / (yk * imw.view(col)).sum(0)
                raw = D * (gy - yk * gw)
                J = raw - yk * raw.sum(0)
                h, _ = gas.enthalpy_cp(ave(bv[5]))
                F[4] = F[4] + (h * J).sum(0)
                for j in range(9):
                    F[5 + j] = J[j]
            _to_dq(dq, F, r, d, 1.0)


def _exact_riemann(dq, case, m, g, jac, met, bv):
    """dq -= differences of the Roe or HLLC face fluxes."""
    nd = 3
    rec, roe = case["recon"], case["scheme"] == 2
    mt = [met[3 * a:3 * a + 3] for a in range(3)]
    if roe:
        cs = [sum((bv[1 + l] * k[l]) for l in range(3)).abs() for k in mt]
        gn = [torch.sqrt((k * k).sum(0)) for k in mt]
        delta = EFIX * (sum(cs) + torch.sqrt(GAM * bv[4] / bv[0]) * sum(gn) / 3)

    def minmod(a, b):
        return torch.where(a * b > 0, torch.sign(a) * torch.minimum(a.abs(), b.abs()), torch.zeros_like(a))

    for d in range(nd):
        for r in _slabs(m, d, 4e6):
            def pt(a, off):
                s = [0, 0, 0]
                s[d] = off
                return _cut(a, g, r, s)

            v = [pt(bv[:5], q) for q in (-1, 0, 1, 2)]
            L, Rr = v[1], v[2]
            if rec > 1:  # both limited forms are the minmod of the two neighbouring differences
                L = v[1] + 0.5 * minmod(v[1] - v[0], v[2] - v[1])
                Rr = v[2] - 0.5 * minmod(v[2] - v[1], v[3] - v[2])
            el, er = [s[4] / (GAM - 1) + 0.5 * s[0] * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2) for s in (L, Rr)]
            kl, kr, jl, jr = pt(mt[d], 0), pt(mt[d], 1), pt(jac, 0), pt(jac, 1)
            k, ja = 0.5 * (kl + kr), 0.5 * (jl + jr)
            gk = torch.sqrt((k * k).sum(0))
            n = k / gk
            sl, sr = torch.sqrt(L[0]), torch.sqrt(Rr[0])
            wl, wr = sl / (sl + sr), sr / (sl + sr)
            u = wl * L[1:4] + wr * Rr[1:4]
            h = wl * (el + L[4]) / L[0] + wr * (er + Rr[4]) / Rr[0]
            ek = 0.5 * (u * u).sum(0)
            c = torch.sqrt((GAM - 1) * (h - ek))
            un = (n * u).sum(0)

            def flux(s, e, kk):
                U = (s[1:4] * kk).sum(0)
                return [s[0] * U] + [s[0] * U * s[1 + l] + s[4] * kk[l] for l in range(3)] + [(e + s[4]) * U]

            if roe:
                fl, fr = flux(L, el, kl * jl), flux(Rr, er, kr * jr)
                fix = 0.5 * (pt(delta, 0) + pt(delta, 1))
                ev = [(x * gk).abs() for x in (un - c, un, un + c)]
                ev = [torch.where(x < fix, 0.5 * (x * x / fix + fix), x) for x in ev]
                dr, dp, du = Rr[0] - L[0], None, None
                w = [ja * dr] + [ja * (Rr[0] * Rr[l] - L[0] * L[l]) for l in (1, 2, 3)] + [ja * (er - el)]
                a1 = (GAM - 1) * (ek * w[0] - sum(u[l] * w[1 + l] for l in range(3)) + w[4]) / (c * c)
                a2 = (sum(n[l] * w[1 + l] for l in range(3)) - un * w[0]) / c
                am, ap, a0 = 0.5 * (a1 - a2) * ev[0], 0.5 * (a1 + a2) * ev[2], (w[0] - a1) * ev[1]
                shear = [(w[1 + l] - u[l] * w[0] - n[l] * a2 * c) * ev[1] for l in range(3)]
                diss = [a0 + am + ap] + [u[l] * (a0 + am + ap) + n[l] * c * (ap - am) + shear[l] for l in range(3)]
                diss.append(ek * a0 + (h - un * c) * am + (h + un * c) * ap + sum(u[l] * shear[l] for l in range(3)))
                F = {q: 0.5 * (fl[q] + fr[q]) - 0.5 * diss[q] for q in range(5)}
            else:
                ul, ur = (n * L[1:4]).sum(0), (n * Rr[1:4]).sum(0)
                cl, cr = torch.sqrt(GAM * L[4] / L[0]), torch.sqrt(GAM * Rr[4] / Rr[0])
                s1, s2 = torch.minimum(ul - cl, un - c), torch.maximum(ur + cr, un + c)
                sm = (Rr[0] * ur * (s2 - ur) - L[0] * ul * (s1 - ul) + L[4] - Rr[4]) / (Rr[0] * (s2 - ur) - L[0] * (s1 - ul))
                pm = L[0] * (s1 - ul) * (sm - ul) + L[4]
                fl, fr = flux(L, el, k), flux(Rr, er, k)
                F = {}
                for q in range(5):
                    star = []
                    for s, e, f, ss, us in ((L, el, fl, s1, ul), (Rr, er, fr, s2, ur)):
                        rs = s[0] * (ss - us) / (ss - sm)
                        if q == 0:
                            x, x0 = rs, s[0]
                        elif q < 4:
                            x, x0 = rs * s[q] + (pm - s[4]) / (ss - sm) * n[q - 1], s[0] * s[q]
                        else:
                            x, x0 = (e * (ss - us) + pm * sm - s[4] * us) / (ss - sm), e
                        star.append(f[q] + ss * gk * (x - x0))
                    f = torch.where(sm >= 0, star[0], star[1])
                    F[q] = ja * torch.where(s1 >= 0, fl[q], torch.where(s2 < 0, fr[q], f))
            _to_dq(dq, F, r, d, -1.0)


def _exact_cv(bv, sv, gas):
    V2 = (bv[1:4] ** 2).sum(0)
    if gas is None:
        return torch.cat([bv[:1], bv[:1] * bv[1:4], (bv[4] / (GAM - 1) + 0.5 * bv[0] * V2)[None]])
    h, _ = gas.enthalpy_cp(bv[5])
    e = bv[0] * ((h * sv).sum(0) + 0.5 * V2) - bv[4]
    return torch.cat([bv[:1], bv[:1] * bv[1:4], e[None], bv[:1] * sv])


def _exact_bc(m, g, wide, cv, bv, sv, gas):
    """Outflow faces of a 2-D block or periodic faces of a 3-D one, over the face's nodes (widened by the ghosts with the
    viscous scheme), then the k ghosts of a 2-D block."""
    state = [bv] if sv is None else [bv, sv]
    e = g if wide else 0

    def face(d, pos):
        s = [slice(g - e, g + n + e) for n in m]
        if m[2] == 1 and not wide:
            s[2] = slice(g, g + 1)
        s[d] = slice(g + pos, g + pos + 1)
        return (Ellipsis, s[2], s[1], s[0])

    def redo(at):
        cv[at] = _exact_cv(bv[at], sv[at] if sv is not None else None, gas)

    for d in range(2 if m[2] == 1 else 3):
        for low in (True, False):
            pos, sgn = (0, -1) if low else (m[d] - 1, 1)
            other = m[d] - 1 - pos
            if m[2] > 1:
                for a in state:
                    mean = 0.5 * (a[face(d, pos)] + a[face(d, other)])
                    a[face(d, pos)] = mean
                    a[face(d, other)] = mean
                redo(face(d, pos))
            for q in range(1, g + 1):
                for a in state:
                    a[face(d, pos + sgn * q)] = a[face(d, (other if m[2] > 1 else pos) + (sgn * q if m[2] > 1 else 0))]
                redo(face(d, pos + sgn * q))
    if m[2] == 1:
        for a in state + [cv]:
            a[..., :, :, :] = a[..., g:g + 1, :, :].clone()


def _exact_step(case, seed):
    gas = None
    if case["kind"] == "air_step":
        g, jac, met, bv, (param, _) = _air_state(case, seed)
        sv = None
    else:
        g, jac, met, bv, sv, (param, _) = _mix_state(case, seed)
        gas = _Gas(_mixture()[0])
    m = (case["mx"], case["my"], case["mz"])
    inner = [(0, n) for n in m]
    viscous, eps = param["viscous_order"] > 0, 1e-40 * param["weno_eps_scale"]
    nd = 3 if m[2] > 1 else 2

    def props():
        if gas:
            return gas.properties(sv, bv[5])
        x = bv[5] / 288.16
        return GAM, torch.sqrt(GAM * R_AIR * bv[5]), 1.7894e-5 * x * torch.sqrt(x) * 398.16 / (bv[5] + 110), None, None

    gam, snd, mu, lam, rd = props()
    cv = _exact_cv(bv, sv, gas)
    gn = [torch.sqrt((met[3 * a:3 * a + 3] ** 2).sum(0)) for a in range(nd)]
    rad = torch.stack([(bv[1:4] * met[3 * a:3 * a + 3]).sum(0).abs() + snd * gn[a] for a in range(nd)]).amax(0)
    if viscous:
        if gas:
            _, cp = gas.enthalpy_cp(bv[5])
            dif = torch.maximum(torch.maximum(mu, lam * gam / (cp * sv).sum(0)), rd.amax(0)) / bv[0]
        else:
            dif = GAM / bv[0] * mu / PR
        rad = torch.maximum(rad, torch.stack(gn).amax(0) ** 2 * dif)
    dt = float((CFL / _cut(rad, g, inner)).min())
    qn = cv.clone()
    J = _cut(jac, g, inner)
    for a, b, c in ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3, 2.0 / 3, 2.0 / 3)):
        dq = torch.zeros((cv.shape[0],) + tuple(J.shape), dtype=F64, device=DEV)
        if viscous:
            _exact_viscous(dq, m, g, jac, met, bv, mu, gas, sv, lam, rd)
        _exact_weno(dq, m, g, case["scheme"], eps, jac, met, cv, bv, gas, snd)
        q = a * _cut(qn, g, inner) + b * _cut(cv, g, inner) + c * dt / J * dq
        if m[2] == 1:
            q[3] = 0
        V = q[1:4] / q[0]
        if gas:
            y = q[5:].clamp(min=0)
            y = y / y.sum(0)
            q[5:] = y * q[0]
            T, R = gas.temperature(y, q[4] / q[0] - 0.5 * (V * V).sum(0), _cut(bv[5], g, inner))
            p = q[0] * R * T
            _cut(sv, g, inner).copy_(y)
        else:
            p = (GAM - 1) * (q[4] - 0.5 * q[0] * (V * V).sum(0))
            T = p / (q[0] * R_AIR)
        _cut(cv, g, inner).copy_(q)
        _cut(bv, g, inner).copy_(torch.cat([q[:1], V, p[None], T[None]]))
        _exact_bc(m, g, param["viscous_order"] == 2, cv, bv, sv, gas)
        gam, snd, mu, lam, rd = props()
    P = jac.numel()
    out = dict(cv=cv.reshape(-1, P), bv=bv.reshape(6, P), mul=mu.reshape(1, P))
    if gas:
        out["sv"] = sv.reshape(9, P)
    return out


def _exact_reactors(case, seed):
    m, s = _reactor_state(case, seed)
    gas = _Gas(m)
    n_sub = torch.floor(DT_REACT / s["reaction_timeScale"]).to(torch.int64)
    order = torch.argsort(n_sub, descending=True)
    n_sub = n_sub[order]
    rho, E = s["cv"][0][order], s["cv"][4][order]
    rY, T, Y = s["cv"][5:][:, order].clone(), s["bv"][5][order].clone(), s["sv"][:, order].clone()
    p, ts = s["bv"][4][order].clone(), s["reaction_timeScale"][order].clone()
    hs = DT_REACT / (n_sub + 1).to(F64)
    sf, sb = [torch.tensor(np.asarray(getattr(m, k), dtype=np.float64), dtype=F64, device=DEV) for k in ("stoi_f", "stoi_b")]
    tb = torch.tensor(np.asarray(m.third_body_coeff), dtype=F64, device=DEV)
    mw = gas.mw[:, None]
    count = torch.bincount(n_sub, minlength=int(n_sub[0]) + 1).flip(0).cumsum(0).flip(0).tolist()
    for step in range(int(n_sub[0]) + 1):
        k = count[step]  # the nodes that still have a substep to take
        t, h = T[:k], hs[:k]
        c = rY[:, :k] / mw * 1e-3
        lnt, it, gb = torch.log(t), 1 / t, gas.gibbs(t)
        make, use = torch.zeros_like(c), torch.zeros_like(c)
        J = torch.zeros((9, 9, k), dtype=F64, device=DEV)
        for r in range(m.n_reac):
            ty = int(m.reac_type[r])
            kf = float(m.A[r]) * torch.exp(float(m.b[r]) * lnt - float(m.Ea[r]) * it)
            low = float(m.A2[r]) * torch.exp(float(m.b2[r]) * lnt - float(m.Ea2[r]) * it)
            cc = (c * tb[r][:, None]).sum(0)
            if ty == 3:
                kf = kf + low
            elif ty == 4:
                kf = kf * cc
            elif ty > 4:
                pr = low * cc / kf
                F = 1.0
                if ty > 5:
                    al = float(m.troe_alpha[r])
                    fc = (1 - al) * torch.exp(-t / float(m.troe_t3[r])) + al * torch.exp(-t / float(m.troe_t1[r]))
                    if ty == 7:
                        fc = fc + torch.exp(-float(m.troe_t2[r]) * it)
                    lf, lp = torch.log10(fc), torch.log10(pr)
                    x = (lp - 0.4 - 0.67 * lf) / (0.75 - 1.27 * lf - 0.14 * (lp - 0.4 - 0.67 * lf))
                    F = 10 ** (lf / (1 + x * x))
                kf = kf * pr / (1 + pr) * F
            q1, q2 = kf, torch.zeros_like(kf)
            if ty != 0:
                kc = (101325.0 / R_U * 1e-3 * it) ** int(m.order[r]) * torch.exp(-((sb[r] - sf[r])[:, None] * gb).sum(0))
                q2 = kf / kc
            for l in range(9):
                q1, q2 = q1 * c[l] ** int(sf[r, l]), q2 * c[l] ** int(sb[r, l])
            inv = [l for l in range(9) if sf[r, l] or sb[r, l]]
            for l in inv:
                make[l] += q2 * sf[r, l] + q1 * sb[r, l]
                use[l] += q1 * sf[r, l] + q2 * sb[r, l]
                net = sb[r, l] - sf[r, l]
                for n in inv:
                    J[l, n] += net * (sf[r, n] * q1 - sb[r, n] * q2)
        w = 1e3 * mw
        rc = torch.where(rY[:, :k] > 1e-25, 1 / rY[:, :k], torch.zeros_like(c))
        A = torch.eye(9, dtype=F64, device=DEV)[:, :, None] - h * J * rc[None] * w[:, None]
        om = torch.linalg.solve(A.permute(2, 0, 1).contiguous(), ((make - use) * w).t().contiguous()).t()
        ud = use * w
        sc = torch.where((rY[:, :k] > 1e-25) & (ud.abs() > 1e-25), (rY[:, :k] / ud).abs(), torch.full_like(c, 1e6))
        ts[:k] = sc.amin(0).clamp(max=1e6)
        x = (rY[:, :k] + om * h).clamp(min=0)
        y = x / x.sum(0)
        rY[:, :k], Y[:, :k] = y * rho[:k], y
        tn, R = gas.temperature(y, E[:k] / rho[:k], t)
        T[:k], p[:k] = tn, rho[:k] * R * tn
    back = torch.argsort(order)
    z = torch.zeros_like(rho)
    cv = torch.cat([torch.stack([rho, z, z, z, E]), rY])[:, back]
    bv = torch.stack([rho, z, z, z, p, T])[:, back]
    return dict(cv=cv, bv=bv, sv=Y[:, back], reaction_timeScale=ts[back])


def _exact_surrogate(case, seed):
    x, gt, w, norm = [a.to(F64) for a in _surrogate_inputs(case, seed)]
    mean, rstd, om, os_, _, _, scale = norm.split((12, 12, 11, 11, 12, 12, 11))
    blocks = [b.view(s) for b, s in zip(w.split((2048, 18432, 18432, 2304)), ((128, 16), (128, 144), (128, 144), (16, 144)))]
    forward = case["kind"] == "surrogate_forward"
    w = [b.clone().requires_grad_(not forward) for b in blocks]
    a = torch.zeros((x.shape[0], 16), dtype=F64, device=DEV)
    a[:, :12], a[:, 15] = (x - mean) * rstd, 1.0
    with torch.set_grad_enabled(not forward):
        for l in range(3):
            h = torch.tanh(a @ w[l].t())
            a = torch.cat([h, torch.ones_like(h[:, :1]), torch.zeros_like(h[:, :15])], 1)
        y = a @ w[3].t()
        if forward:
            return y
        z = torch.where(scale > 0, torch.asinh(gt / torch.where(scale > 0, scale, 1.0)), gt)
        loss = ((y[:, :11] - (z - om) / os_) ** 2).mean()
        loss.backward()
    return {"loss": float(loss.detach()), "grad": torch.cat([b.grad.reshape(-1) for b in w])}


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("surrogate"):
        return _exact_surrogate(case, seed)
    if kind == "reactors":
        return _exact_reactors(case, seed)
    if kind in ("air_step", "mix_step"):
        return _exact_step(case, seed)
    m = (case["mx"], case["my"], case["mz"])
    gas = sv = None
    if kind.startswith("air"):
        g, jac, met, bv, (param, _) = _air_state(case, seed)
        x = bv[5] / 288.16
        mu, snd, lam, rd = 1.7894e-5 * x * torch.sqrt(x) * 398.16 / (bv[5] + 110), None, None, None
    else:
        g, jac, met, bv, sv, (param, _) = _mix_state(case, seed)
        gas = _Gas(_mixture()[0])
        _, snd, mu, lam, rd = gas.properties(sv, bv[5])
    dq = torch.zeros((param["n_var"], m[2], m[1], m[0]), dtype=F64, device=DEV)
    if kind.endswith("viscous"):
        _exact_viscous(dq, m, g, jac, met, bv, mu, gas, sv, lam, rd)
    elif kind == "air_riemann":
        _exact_riemann(dq, case, m, g, jac, met, bv)
    else:
        _exact_weno(dq, m, g, case["scheme"], 1e-40 * param["weno_eps_scale"], jac, met, _exact_cv(bv, sv, gas), bv, gas, snd)
    return dq.reshape(param["n_var"], -1)

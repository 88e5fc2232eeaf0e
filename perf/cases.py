"""The work that programs have this library do, as cases that can be timed.

A case is one call sequence of a user's program through the public entry points
(`Device`, `Ensemble`, `autograd`), over the sizes, precisions and options that
such programs use:

* ``step``        k whole RK3 steps (acDeviceIntegrateStep), then the fields into a
                  torch tensor, as a run that looks at its state every k steps;
* ``loop``        the same through the reference's own calls: boundconds, substep,
                  swap, three times a step;
* ``turbulence``  forced turbulence: upwinding and helical forcing, through the loop;
* ``adaptive``    steps whose dt comes from the on-device CFL maxima of the last one;
* ``diagnostics`` the scalar and vector reductions that a run prints;
* ``ensemble``    k steps of many small independent meshes, then every member's fields;
* ``gradient``    final-time energy of k steps and its gradient (forward and backward).

Initial fields follow the seeded distributions of the benchmark workloads: small
uniform lnrho and entropy, Gaussian velocity and vector potential, on [0, 2 pi)^3.
``exact`` is the same mathematics in plain FP64 torch.
"""
import math

import numpy as np
import torch

G = 3  # ghost cells per side
NF = 8

NU = ETA = 5e-3
GAMMA, CP, CS, LNT0, LNRHO0, MU0, ZETA, K_HEAT = 5.0 / 3.0, 1.0, 1.0, 1.2, 1.3, 1.4, 0.01, 1e-3

# A helical force on the k = (1, 1, 1) mode: re and im are perpendicular to k.
FORCE = dict(magnitude=1e-4, phase=0.9, kaver=math.sqrt(3.0), k=(1.0, 1.0, 1.0),
             re=(0.5 / math.sqrt(2.0), -0.5 / math.sqrt(2.0), 0.0),
             im=(1.0 / math.sqrt(6.0), 1.0 / math.sqrt(6.0), -2.0 / math.sqrt(6.0)))

ENSEMBLE_SIZES = (32, 48, 64, 96)


def case(name, kind, nx, ny=None, nz=None, precision=0, steps=1, **more):
    return dict(name=name, kind=kind, nx=nx, ny=ny or nx, nz=nz or nx, precision=precision,
                steps=steps, **more)


def listed():
    return [
        # the smallest mesh of the smoke test and of the ensemble: launches count
        case("step_fp64_32", "step", 32, steps=20),
        # the 128^3 FP64 parity workload
        case("step_fp64_128", "step", 128, steps=10),
        # the headline: 512^3 FP64, state resident in HBM
        case("step_fp64_512", "step", 512, steps=2),
        # FP32-compensated runs: an ordinary and the largest mesh
        case("step_fp32c_256", "step", 256, precision=1, steps=5),
        case("step_fp32c_512", "step", 512, precision=1, steps=2),
        # a box whose sides are no multiples of a tile, through the reference's calls
        case("loop_fp64_ragged", "loop", 150, 101, 67, steps=10),
        # an odd side along x (rows that are no multiple of 16 bytes)
        case("loop_fp64_odd", "loop", 125, 125, 125, steps=5),
        # forced turbulence with upwinding, as the subsonic turbulence setup of the reference
        case("turbulence_fp64_128", "turbulence", 128, steps=5),
        # adaptive timestep: one host read of the CFL maxima per step
        case("adaptive_fp32c_256", "adaptive", 256, precision=1, steps=4),
        # the printed diagnostics of an ordinary FP64 run
        case("diagnostics_fp64_256", "diagnostics", 256),
        # parameter study: many small FP32-compensated meshes on one GPU
        case("ensemble_fp32c_32", "ensemble", 32, precision=1, steps=40, members=32),
        # gradient of the final energy with respect to the initial fields, nu and eta
        case("gradient_fp64_64", "gradient", 64, steps=10, every=5),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step"] * 4 + ["loop"] * 3 + ["turbulence", "turbulence", "adaptive",
                                                     "adaptive", "diagnostics", "ensemble",
                                                     "gradient"])
    precision = rng.randrange(2)
    if kind == "ensemble":
        m = rng.randrange(4, 33)
        return dict(kind=kind, nx=32, ny=32, nz=32, precision=precision,
                    steps=rng.randrange(5, 41), members=m)
    if kind == "gradient":
        every = rng.randrange(2, 6)
        return dict(kind=kind, nx=side(16, 96), ny=side(16, 80), nz=side(16, 80),
                    precision=precision, steps=rng.randrange(2, 11), every=every)
    hi = 256 if kind in ("turbulence", "adaptive") else 400
    n = [side(24, hi) for _ in range(3)]
    if rng.random() < 0.3:  # cubic meshes are common
        n = [n[0]] * 3
    if rng.random() < 0.6:  # and so are even sides along x
        n[0] += n[0] & 1
    cells = n[0] * n[1] * n[2]
    steps = 1 if kind == "diagnostics" else max(1, min(rng.randrange(1, 21), int(2.5e8 // cells)))
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], precision=precision, steps=steps)


# ---- inputs ----


def _fields(c, seed, shape=None):
    """The initial fields (8, nz, ny, nx) on the GPU, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = shape or (c["nz"], c["ny"], c["nx"])
    f = torch.empty((NF, *shape), dtype=torch.float64, device="cuda")
    # developed turbulence has larger amplitudes than the noise that runs start from
    amp = 1e-2 if c["kind"] in ("turbulence", "adaptive", "diagnostics") else 1e-5
    f[0].uniform_(-amp, amp, generator=g)
    f[1:4].normal_(0.0, 3e-2 if amp == 1e-2 else 1e-3, generator=g)
    f[4:7].normal_(0.0, 3e-3 if amp == 1e-2 else 1e-4, generator=g)
    f[7].uniform_(-amp, amp, generator=g)
    return f


def _mesh(f):
    """(8, nz, ny, nx) with zero ghost zones around, as a host or device mesh has."""
    m = torch.zeros((NF, *(s + 2 * G for s in f.shape[1:])), dtype=torch.float64, device="cuda")
    _inner(m).copy_(f)
    return m


def _inner(m):
    return m[..., G:-G, G:-G, G:-G]


def _dt(c):
    # explicit diffusion at (4/3 nu + zeta) and sound waves, well inside RK3's limits
    ds = min(2 * math.pi / n for n in (c["nx"], c["ny"], c["nz"]))
    return min(1e-3, 1.6 * ds * ds / (18.13 * (4.0 / 3.0 * NU + ZETA)))


def _info(c):
    from astaroth_b200 import capi
    from astaroth_b200.device import CONFIG_PARAMS, make_info

    more = {}
    if c["kind"] == "turbulence":
        more = dict(upwind=1, current_time=1.0, forcing_magnitude=FORCE["magnitude"],
                    forcing_phase=FORCE["phase"], kaver=FORCE["kaver"])
        for a, x in enumerate("xyz"):
            more["k_force" + x] = FORCE["k"][a]
            more["ff_hel_re" + x] = FORCE["re"][a]
            more["ff_hel_im" + x] = FORCE["im"][a]
    if c["kind"] == "adaptive":
        # the stable diffusive factor of the 6th-order Laplacian, and an advective bound below
        # it, so that dt changes from step to step
        more = dict(cdtv=0.04, cdt=0.2)
    info = make_info((c["nx"], c["ny"], c["nz"]), precision=c["precision"],
                     **dict(CONFIG_PARAMS, **more))
    if c["kind"] == "turbulence":
        info.int_params[capi.IntParam.AC_lforcing] = 1
    return info


def _members(c):
    """Side, nu, eta of every member of an ensemble: the same study for every seed."""
    rng = np.random.default_rng(3)
    m = c["members"]
    ns = rng.choice(np.asarray(ENSEMBLE_SIZES), size=m)
    nus, etas = 10.0 ** rng.uniform(-3.0, -2.0, size=m), 10.0 ** rng.uniform(-3.0, -2.0, size=m)
    return [(int(n), float(a), float(b)) for n, a, b in zip(ns, nus, etas)]


def prepare(c, seed):
    from astaroth_b200.device import CONFIG_PARAMS, Device, make_info

    if c["kind"] == "ensemble":
        from astaroth_b200.ensemble import Ensemble

        members = _members(c)
        e = Ensemble([make_info(n, precision=c["precision"],
                                **dict(CONFIG_PARAMS, nu_visc=nu, eta=eta))
                      for n, nu, eta in members])
        # the form that the autotuner finds for these sizes (tiled launches in graph branches)
        e.set_tiles(32, 4, 8, 0, 1)
        e.set_timesteps(1e-3)
        out = []
        for m, (n, _, _) in enumerate(members):
            mesh = _mesh(_fields(c, seed * 1000 + m, (n, n, n)))
            e.load_member(m, mesh.cpu().numpy())
            # page-locked result arrays, kept by the program
            out.append(torch.empty(mesh.shape, dtype=torch.float64, pin_memory=True).numpy())
        return dict(case=c, ensemble=e, out=out)
    info = _info(c)
    dev = Device(info)
    f0 = _mesh(_fields(c, seed))
    if c["kind"] == "gradient":
        return dict(case=c, dev=dev, info=info, f0=f0.requires_grad_(), dt=_dt(c),
                    nu=torch.tensor(NU, dtype=torch.float64, device="cuda", requires_grad=True),
                    eta=torch.tensor(ETA, dtype=torch.float64, device="cuda", requires_grad=True))
    dev.load_mesh_device(f0)
    dev.synchronize()
    if c["kind"] == "diagnostics":
        return dict(case=c, dev=dev)
    if c["kind"] == "adaptive":
        dev.periodic_boundconds()
        dev.calc_timestep()
    return dict(case=c, dev=dev, dt=_dt(c), out=torch.empty_like(f0))


# ---- one pass ----


def run(state):
    c = state["case"]
    if c["kind"] == "ensemble":
        e = state["ensemble"]
        for _ in range(c["steps"]):
            e.integrate_step()
        return [_inner(e.store_member(m, out)) for m, out in enumerate(state["out"])]
    dev = state["dev"]
    if c["kind"] == "gradient":
        from astaroth_b200 import autograd

        f = autograd.integrate(state["f0"], state["nu"], state["eta"], dev, c["steps"],
                               state["dt"], checkpoint_every=c["every"])
        energy = autograd.energy(f, state["info"])
        g, gnu, geta = torch.autograd.grad(energy, (state["f0"], state["nu"], state["eta"]))
        return [energy.detach(), gnu, geta] + list(_inner(g))
    if c["kind"] == "diagnostics":
        dev.periodic_boundconds()
        got = {"umax": dev.reduce_vec("RTYPE_MAX", 1, 2, 3),
               "urms": dev.reduce_vec("RTYPE_RMS", 1, 2, 3),
               "arms": dev.reduce_vec("RTYPE_RMS", 4, 5, 6),
               "rho": dev.reduce_scal("RTYPE_RMS_EXP", 0),
               "alfven": dev.reduce_vec_scal("RTYPE_ALFVEN_RMS", 4, 5, 6, 0)}
        for q in range(NF):
            got["max%d" % q] = dev.reduce_scal("RTYPE_MAX", q)
            got["min%d" % q] = dev.reduce_scal("RTYPE_MIN", q)
            got["rms%d" % q] = dev.reduce_scal("RTYPE_RMS", q)
        dev.calc_timestep()
        got["dt"] = dev.timestep()
        return got
    for _ in range(c["steps"]):
        if c["kind"] == "adaptive":
            dev.integrate_step(dev.timestep())
        elif c["kind"] == "step":
            dev.integrate_step(state["dt"])
        else:
            dev.integrate_step_loop(state["dt"])
    return list(_inner(dev.store_mesh_device(state["out"])))


# ---- what a pass cannot do without ----


def work(c):
    cells = c["nx"] * c["ny"] * c["nz"]
    # per cell: one RK3 step reads each field 5 times and writes it 3 times (2N scheme with
    # the previous state; FP32-compensated values are 8-byte pairs); a right-hand side is
    # 24 axial first and second derivatives (16 operations), 12 mixed ones (14), and about
    # 250 operations of the equations; the update is 6 per field
    step_bytes, step_flops = 512.0, 3 * (24 * 16 + 12 * 14 + 250 + 48.0)
    if c["kind"] == "ensemble":
        cells = sum(n ** 3 for n, _, _ in _members(c))
        return dict(bytes=cells * (step_bytes * c["steps"] + 128), flops=cells * step_flops * c["steps"])
    if c["kind"] == "gradient":
        # forward, recomputed forward, and a reverse sweep that reads the state and the two
        # adjoints and writes the two adjoints, with about three times the operations
        n = c["steps"]
        return dict(bytes=cells * n * (2 * step_bytes + 3 * 5 * 64.0),
                    flops=cells * n * 5 * step_flops)
    if c["kind"] == "diagnostics":
        # 24 one-field, 3 three-field reductions, one of four fields, exp(lnrho), and dt
        return dict(bytes=cells * 8.0 * (24 + 9 + 4 + 1 + 7), flops=cells * 150.0)
    return dict(bytes=cells * (step_bytes * c["steps"] + 128), flops=cells * step_flops * c["steps"])


def tolerance(c):
    # measured against exact(), which sums in another order.  FP64 fields: up to 6e-16 after
    # 20 steps; gradients 7e-15 (the sums over all cells for nu and eta).  FP32-compensated:
    # rates in FP32 on a 48-bit state, up to 1.5e-7; its FP64 reverse sweep is about states
    # that are off by that much: 1e-9 to 1e-8.
    if c["kind"] == "gradient":
        return {"rel": 4e-14, "max": 1e-12} if c["precision"] == 0 else {"rel": 4e-8, "max": 2e-6}
    if c["kind"] == "diagnostics":
        return {"rel": 1e-14} if c["precision"] == 0 else {"rel": 6e-7}
    return {"rel": 3e-15, "max": 2e-13} if c["precision"] == 0 else {"rel": 6e-7, "max": 3e-5}


# ---- the same in plain FP64 torch ----

_C1 = (3 / 4, -3 / 20, 1 / 60)
_C2 = (-49 / 18, 3 / 2, -3 / 20, 1 / 90)
_CM = (270 / 720, -27 / 720, 2 / 720)
_CU = (-20 / 60, 15 / 60, -6 / 60, 1 / 60)
_ALPHA = (0.0, -5.0 / 9.0, -153.0 / 128.0)
_BETA = (1.0 / 3.0, 15.0 / 16.0, 8.0 / 15.0)


def _pad(f, z0=0, z1=None):
    """Periodic ghost zones around planes z0..z1 of (..., nz, ny, nx)."""
    nz = f.shape[-3]
    z = torch.arange(z0 - G, (nz if z1 is None else z1) + G, device=f.device) % nz
    p = f.index_select(f.dim() - 3, z)
    for d in (-1, -2):
        n = p.shape[d]
        i = torch.arange(-G, n + G, device=f.device) % n
        p = p.index_select(p.dim() + d, i)
    return p


def _rates(p, inv, nu, eta, upwind=False):
    """Rates of the 8 fields from the list p of padded fields (..., z, y, x); nu and eta may be
    tensors that broadcast against a field."""
    n = [p[0].shape[-1 - a] - 2 * G for a in range(3)]

    def at(f, dx, dy, dz):
        return f[..., G + dz:G + dz + n[2], G + dy:G + dy + n[1], G + dx:G + dx + n[0]]

    def on(f, a, k):
        return at(f, *(k if a == b else 0 for b in range(3)))

    def d1(f, a):
        return sum(c * (on(f, a, k) - on(f, a, -k)) for k, c in enumerate(_C1, 1)) * inv[a]

    def d2(f, a):
        r = _C2[0] * on(f, a, 0)
        for k in (1, 2, 3):
            r = r + _C2[k] * (on(f, a, k) + on(f, a, -k))
        return r * inv[a] ** 2

    def up(f, a):
        r = _CU[0] * on(f, a, 0)
        for k in (1, 2, 3):
            r = r + _CU[k] * (on(f, a, k) + on(f, a, -k))
        return r * inv[a]

    def mix(f, a, b):
        r = 0
        for k, c in enumerate(_CM, 1):
            o = [[0, 0, 0] for _ in range(4)]
            for w, (s, t) in enumerate(((k, k), (-k, -k), (k, -k), (-k, k))):
                o[w][a], o[w][b] = s, t
            r = r + c * ((at(f, *o[0]) + at(f, *o[1])) - (at(f, *o[2]) + at(f, *o[3])))
        return r * (inv[a] * inv[b])

    def grad(f):
        return [d1(f, a) for a in range(3)]

    def vector(v):
        g = [grad(f) for f in v]
        dd = [[d2(f, a) for a in range(3)] for f in v]
        lap = [sum(d) for d in dd]
        gd = [dd[0][0] + mix(v[1], 0, 1) + mix(v[2], 0, 2),
              mix(v[0], 0, 1) + dd[1][1] + mix(v[2], 1, 2),
              mix(v[0], 0, 2) + mix(v[1], 1, 2) + dd[2][2]]
        return g, lap, gd

    lnrho, s = at(p[0], 0, 0, 0), at(p[7], 0, 0, 0)
    u = [at(f, 0, 0, 0) for f in p[1:4]]
    gl, gs = grad(p[0]), grad(p[7])
    lapl, laps = sum(d2(p[0], a) for a in range(3)), sum(d2(p[7], a) for a in range(3))
    gu, lapu, gdu = vector(p[1:4])
    ga, lapa, gda = vector(p[4:7])
    divu = gu[0][0] + gu[1][1] + gu[2][2]
    b = [ga[2][1] - ga[1][2], ga[0][2] - ga[2][0], ga[1][0] - ga[0][1]]
    j = [(gda[a] - lapa[a]) / MU0 for a in range(3)]
    e = torch.exp(GAMMA * s / CP + (GAMMA - 1) * (lnrho - LNRHO0))
    irho = torch.exp(-lnrho)
    st = [[0.5 * (gu[a][c] + gu[c][a]) - (divu / 3 if a == c else 0) for c in range(3)]
          for a in range(3)]
    ss = sum(st[a][c] ** 2 for a in range(3) for c in range(3))
    jxb = [j[1] * b[2] - j[2] * b[1], j[2] * b[0] - j[0] * b[2], j[0] * b[1] - j[1] * b[0]]
    r = [-(u[0] * gl[0] + u[1] * gl[1] + u[2] * gl[2]) - divu]
    for c in range(3):
        r.append(-(u[0] * gu[c][0] + u[1] * gu[c][1] + u[2] * gu[c][2])
                 - CS * CS * e * (gs[c] / CP + gl[c]) + irho * jxb[c]
                 + nu * (lapu[c] + gdu[c] / 3
                         + 2 * (st[c][0] * gl[0] + st[c][1] * gl[1] + st[c][2] * gl[2]))
                 + ZETA * gdu[c])
    if upwind:
        au = [abs(x) for x in u]
        for q in range(4):
            r[q] = r[q] + sum(au[a] * up(p[q], a) for a in range(3))
    r += [u[1] * b[2] - u[2] * b[1] + eta * lapa[0], u[2] * b[0] - u[0] * b[2] + eta * lapa[1],
          u[0] * b[1] - u[1] * b[0] + eta * lapa[2]]
    heating = (irho * eta * MU0 * (j[0] ** 2 + j[1] ** 2 + j[2] ** 2) + 2 * nu * ss
               + ZETA * divu * divu) / (math.exp(LNT0) * e)
    sec = [GAMMA / CP * gs[a] + (GAMMA - 1) * gl[a] for a in range(3)]
    first = GAMMA / CP * laps + (GAMMA - 1) * lapl
    heat = K_HEAT * irho * (first + sec[0] ** 2 + sec[1] ** 2 + sec[2] ** 2)
    r.append(-(u[0] * gs[0] + u[1] * gs[1] + u[2] * gs[2]) + heating + heat)
    return r, b, irho


def _inv_ds(c):
    return [c[k] / (2 * math.pi) for k in ("nx", "ny", "nz")]


def _force(c, dt, device):
    """The helical force added to u at the end of a step."""
    x = [torch.arange(c[k], device=device, dtype=torch.float64) * (FORCE["k"][a] * 2 * math.pi / c[k])
         for a, k in enumerate(("nx", "ny", "nz"))]
    ph = x[2][:, None, None] + x[1][None, :, None] + x[0][None, None, :] + FORCE["phase"]
    scale = math.sqrt(dt) * CS * FORCE["magnitude"] * math.sqrt(FORCE["kaver"] * CS)
    return [scale * (FORCE["re"][a] * torch.cos(ph) - FORCE["im"][a] * torch.sin(ph))
            for a in range(3)]


def _substep(f, w, s, dt, inv, nu, eta, upwind=False):
    """(f, w) after substep s, in place on w, in slabs of planes; f is replaced."""
    nz = f.shape[-3]
    zc = max(1, int(3e7 // (f[0, ..., 0, :, :].numel())))
    new = torch.empty_like(f)
    for z0 in range(0, nz, zc):
        z1 = min(nz, z0 + zc)
        r, _, _ = _rates(list(_pad(f, z0, z1)), inv, nu, eta, upwind)
        for q in range(NF):
            v = w[q][..., z0:z1, :, :]
            v.mul_(_ALPHA[s]).add_(r[q], alpha=dt) if s else v.copy_(dt * r[q])
            new[q][..., z0:z1, :, :] = f[q][..., z0:z1, :, :] + _BETA[s] * v
    return new


def _max_speeds(c, f, inv):
    """max |u| and max sqrt(B^2 / rho)."""
    p = list(_pad(f))
    u2 = f[1] ** 2 + f[2] ** 2 + f[3] ** 2
    _, b, irho = _rates(p, inv, NU, ETA)
    va2 = (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) * irho
    return math.sqrt(float(u2.max())), math.sqrt(float(va2.max()))


def _cfl_dt(c, umax, vamax, cdt=0.2, cdtv=0.04):
    ds = min(2 * math.pi / n for n in (c["nx"], c["ny"], c["nz"]))
    adv = cdt * ds / (umax + math.sqrt(CS * CS + vamax * vamax))
    return min(adv, cdtv * ds * ds / max(NU, ETA))


def _exact_gradient(c, f0):
    from torch.utils.checkpoint import checkpoint

    inv, dt = _inv_ds(c), _dt(c)
    f0 = f0.requires_grad_()
    nu = torch.tensor(NU, dtype=torch.float64, device="cuda", requires_grad=True)
    eta = torch.tensor(ETA, dtype=torch.float64, device="cuda", requires_grad=True)

    def sub(f, w, s, nu, eta):
        r = torch.stack(_rates(list(_pad(f)), inv, nu, eta)[0])
        w = _ALPHA[s] * w + dt * r
        return f + _BETA[s] * w, w

    f, w = f0, torch.zeros_like(f0)
    for _ in range(c["steps"]):
        for s in range(3):
            f, w = checkpoint(sub, f, w, s, nu, eta, use_reentrant=False)
    p = list(_pad(f))
    dv = 1.0 / (inv[0] * inv[1] * inv[2])
    _, b, _ = _rates(p, inv, nu.detach(), eta.detach())
    kin = 0.5 * torch.exp(f[0]) * (f[1] ** 2 + f[2] ** 2 + f[3] ** 2)
    energy = ((kin + (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) / (2 * MU0)) * dv).sum()
    g, gnu, geta = torch.autograd.grad(energy, (f0, nu, eta))
    return [energy.detach(), gnu, geta] + list(g)


def _exact_ensemble(c, seed):
    members = _members(c)
    out = [None] * len(members)
    for n in sorted({m[0] for m in members}):  # members of one size together
        who = [i for i, m in enumerate(members) if m[0] == n]
        f = torch.stack([_fields(c, seed * 1000 + i, (n, n, n)) for i in who], dim=1)
        nu, eta = (torch.tensor([members[i][k] for i in who], dtype=torch.float64,
                                device="cuda")[:, None, None, None] for k in (1, 2))
        w = torch.empty_like(f)
        for _ in range(c["steps"]):
            for s in range(3):
                f = _substep(f, w, s, 1e-3, [n / (2 * math.pi)] * 3, nu, eta)
        for i, m in enumerate(who):
            out[m] = f[:, i].cpu().numpy()
    return out


def exact(c, seed):
    if c["kind"] == "ensemble":
        # some 20 ms a step: the smaller ones only
        return _exact_ensemble(c, seed) if c["steps"] * c["members"] <= 1300 else None
    f = _fields(c, seed)
    inv = _inv_ds(c)
    if c["kind"] == "gradient":
        return _exact_gradient(c, f)
    if c["kind"] == "diagnostics":
        rms = lambda t: math.sqrt(float(t.square().mean()))  # noqa: E731
        u2 = f[1] ** 2 + f[2] ** 2 + f[3] ** 2
        a2 = f[4] ** 2 + f[5] ** 2 + f[6] ** 2
        # RTYPE_ALFVEN_RMS maps |v|^2 / exp(scalar)
        got = {"umax": math.sqrt(float(u2.max())), "urms": math.sqrt(float(u2.mean())),
               "arms": math.sqrt(float(a2.mean())), "rho": rms(torch.exp(f[0])),
               "alfven": math.sqrt(float((a2 / torch.exp(f[0])).mean()))}
        for q in range(NF):
            got["max%d" % q], got["min%d" % q] = float(f[q].max()), float(f[q].min())
            got["rms%d" % q] = rms(f[q])
        got["dt"] = _cfl_dt(c, *_max_speeds(c, f, inv), cdt=0.4, cdtv=0.3)
        return got
    dt, w = _dt(c), torch.empty_like(f)
    if c["kind"] == "adaptive":
        dt = _cfl_dt(c, *_max_speeds(c, f, inv))
    force = _force(c, dt, f.device) if c["kind"] == "turbulence" else None
    for _ in range(c["steps"]):
        here = dt
        for s in range(3):
            if s == 2 and c["kind"] == "adaptive":  # the next step's dt
                dt = _cfl_dt(c, *_max_speeds(c, f, inv))
            f = _substep(f, w, s, here, inv, NU, ETA, c["kind"] == "turbulence")
        if force:
            for a in range(3):
                f[1 + a] += force[a]
    return list(f)

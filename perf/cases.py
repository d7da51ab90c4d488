"""What this framework is used for, as cases whose speed can be measured.

Three kinds of pass, all through the public entry points:

- ``step``: one ``Model.evolve_once`` (the reference's ``Solver::evolve_once``), the work
  of every simulation.  Set-ups: the Sedov-Taylor blast, the homogeneous box of the
  reference's throughput benchmark (varying Cullen & Dehnen viscosity, dt = 0 as its
  ``set_next_dt(0.0)``), the clustered box (uneven neighbour counts), the Keplerian disc
  (locally isothermal, point mass, free boundary) and the travelling sound wave (runs in
  the compensated tier).  Precisions: ``mixed`` (error-controlled) and ``fp64`` (the
  default of ``SolverConfig``).
- ``rollout``: ``adjoint.rollout`` over a few steps and its backward pass, as an
  optimisation over initial velocities, energies and the viscosity runs it.
- ``modules``: the module-level chain a host solver calls: tree, neighbour cache,
  h iteration, Omega, equation of state, derivatives.

Sizes: a state of 2,048 particles (launches and latency), the 131,072- and
1,048,576-particle Sedov set-ups of the benchmark, ragged particle counts, and up to
the 8.4-million-particle homogeneous box of the reference's published runs.
"""

import math

import torch

import shamrock_gb300 as sg
from shamrock_gb300 import adjoint, modules
from shamrock_gb300 import _lib as L

HFACT = 1.2
NEIGHBOURS = 58  # M4 kernel at hfact 1.2: 4/3 pi (2 hfact)^3
FIELDS = ("xyz", "vxyz", "axyz", "hpart", "uint", "duint", "omega")


# ------------------------------------------------------------------------ the cases
def listed():
    return [
        # a small test problem or the early iterations of a convergence study: launches
        # and host latency count
        dict(name="sedov_2k_mixed", kind="step", setup="sedov", size=8, precision="mixed"),
        # the first benchmark configuration's size
        dict(name="sedov_131k_mixed", kind="step", setup="sedov", size=32, precision="mixed"),
        # the default workload of the benchmark
        dict(name="sedov_1m_mixed", kind="step", setup="sedov", size=64, precision="mixed"),
        # the reference's own throughput benchmark, at the size of its published CPU runs
        dict(name="homogeneous_8m_mixed", kind="step", setup="homogeneous", size=1 << 23,
             precision="mixed"),
        # uneven density: a clump 100 times denser than the background, a ragged count
        dict(name="clustered_3m_mixed", kind="step", setup="clustered", size=3000017,
             precision="mixed"),
        # accretion disc around a point mass, free boundary, locally isothermal
        dict(name="disc_1m_mixed", kind="step", setup="disc", size=1000003, precision="mixed"),
        # smooth flow on a large background pressure: every step in the compensated tier
        dict(name="soundwave_262k_mixed", kind="step", setup="soundwave", size=64,
             precision="mixed"),
        # the default precision: bit-identical to the FP64 reference path
        dict(name="sedov_131k_fp64", kind="step", setup="sedov", size=32, precision="fp64"),
        # the default precision with the varying viscosity
        dict(name="homogeneous_131k_fp64", kind="step", setup="homogeneous", size=1 << 17,
             precision="fp64"),
        # gradients of a final-state loss: the differentiable sound wave
        dict(name="rollout_soundwave_262k", kind="rollout", setup="soundwave", size=64,
             precision="mixed", steps=5),
        # gradients of the disc's kinetic energy, a ragged count, two segments
        dict(name="rollout_disc_300k", kind="rollout", setup="disc", size=300007,
             precision="mixed", steps=4),
        # a host solver that calls the modules one by one
        dict(name="modules_120k_fp64", kind="modules", setup="clustered", size=120011,
             precision="fp64"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "step", "rollout", "modules"])
    if kind == "modules":
        return dict(kind=kind, setup="clustered", size=log_int(3000, 120000),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "rollout":
        setup = rng.choice(["soundwave", "disc", "sedov"])
        size = {"soundwave": log_int(16, 60), "disc": log_int(5000, 280000),
                "sedov": log_int(8, 38)}[setup]
        return dict(kind=kind, setup=setup, size=size, precision="mixed",
                    steps=rng.randint(2, 5), jitter=round(rng.uniform(0.02, 0.08), 4))
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    setup = rng.choice(["sedov", "sedov", "homogeneous", "clustered", "disc", "soundwave"])
    if precision == "fp64":
        size = {"sedov": log_int(8, 32), "soundwave": log_int(12, 50)}.get(
            setup, log_int(2000, 125000))
    else:
        size = {"sedov": log_int(8, 90), "soundwave": log_int(12, 96)}.get(
            setup, log_int(2000, 3000000))
    case = dict(kind=kind, setup=setup, size=size, precision=precision)
    if setup == "sedov":
        case["jitter"] = round(rng.uniform(0.02, 0.08), 4)
    return case


# ------------------------------------------------------------------------ the set-ups
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _grid(nx, ny, nz):
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) for n in (nx, ny, nz)]
    return torch.stack([t.reshape(-1) for t in torch.meshgrid(*ax, indexing="ij")])


def _sedov(size, g, jitter=0.05):
    """4 size^3 particles on an FCC lattice with position jitter (a fraction of the cell),
    E = 1 injected within two cells of the centre (the jittered benchmark set-up)."""
    basis = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]],
                         device="cuda", dtype=torch.float64) + 0.25
    pos = (_grid(size, size, size)[:, :, None] + basis.T[:, None, :]).reshape(3, -1) / size
    n = pos.shape[1]
    pos = torch.remainder(pos + (jitter / size) * _normal(g, 3, n), 1.0)
    u = torch.full((n,), 1e-5, device="cuda", dtype=torch.float64)
    inside = (pos - 0.5).square().sum(0).sqrt() < 2.0 / size
    u[inside] += n / inside.sum()
    return dict(pos=pos, vel=torch.zeros_like(pos), u=u, gamma=5.0 / 3.0, pmass=1.0 / n,
                h=torch.full_like(u, HFACT * (1.0 / n) ** (1.0 / 3.0)), alpha=1.0, cfl=0.3,
                box=((0.0,) * 3, (1.0,) * 3), periodic=True)


def _homogeneous(size, g):
    """About ``size`` particles on the HCP lattice that closes a periodic box of side near
    1.2, rho = 1, a central energy injection, and a seeded 1 % lattice noise."""
    dr = (0.74 * (1.2**3 / size) / ((4.0 / 3.0) * math.pi)) ** (1.0 / 3.0)
    s = (2.0, math.sqrt(3.0), 2.0 * math.sqrt(6.0) / 3.0)
    nx, ny, nz = (max(4, 2 * int(round(0.6 / (dr * t)))) for t in s)
    i, j, k = _grid(nx, ny, nz)
    box = torch.tensor([s[0] * nx, s[1] * ny, s[2] * nz], device="cuda",
                       dtype=torch.float64) * dr
    pos = torch.stack([s[0] * i + torch.remainder(j + k, 2.0),
                       s[1] * (j + torch.remainder(k, 2.0) / 3.0), s[2] * k]) * dr
    n = pos.shape[1]
    pos = torch.remainder(pos + 0.01 * dr * _normal(g, 3, n), box[:, None])
    q = (pos - 0.5 * box[:, None]).square().sum(0).sqrt() / (16 * dr)
    f = torch.where(q < 1, 0.25 * (2 - q) ** 3 - (1 - q) ** 3,
                    0.25 * (2 - q).clamp(min=0.0) ** 3)
    hi = tuple(box.tolist())
    return dict(pos=pos, vel=torch.zeros_like(pos), u=f / (math.pi * (16 * dr) ** 3),
                gamma=5.0 / 3.0, pmass=hi[0] * hi[1] * hi[2] / n,
                h=torch.full((n,), HFACT * (hi[0] * hi[1] * hi[2] / n) ** (1.0 / 3.0),
                             device="cuda", dtype=torch.float64),
                av="cd10", alpha=0.0, cfl=0.1, dt_zero=True, box=((0.0,) * 3, hi), periodic=True)


def _jittered(side, g):
    p = (_grid(side, side, side) + 0.5) / side
    return p + (0.1 / side) * _normal(g, *p.shape)


def _clustered(size, g, sigma=0.05):
    """Half the particles uniform in the unit cube, half in a Gaussian clump of width sigma,
    both from jittered lattices (the clump by radial stretch mapping)."""
    n1, n2 = size // 2, size - size // 2
    p1 = _jittered(int(math.ceil(n1 ** (1.0 / 3.0))), g)
    keep = torch.argsort(_uniform(g, p1.shape[1]))[:n1]
    p1 = torch.remainder(p1[:, keep], 1.0)
    q = _jittered(int(math.ceil((n2 * 6.0 / math.pi) ** (1.0 / 3.0))) + 2, g) * 2.0 - 1.0
    rq = q.square().sum(0).sqrt()
    keep = torch.argsort(rq)[:n2]
    q, rq = q[:, keep], rq[keep]
    frac = (rq / rq.max()) ** 3 * (1.0 - 1e-9)
    r = torch.linspace(0.0, 8.0, 4096, device="cuda", dtype=torch.float64)
    cdf = torch.erf(r / math.sqrt(2.0)) - math.sqrt(2.0 / math.pi) * r * torch.exp(-0.5 * r * r)
    at = torch.searchsorted(cdf, frac).clamp(1, 4095)
    c0, c1 = cdf[at - 1], cdf[at]
    new = sigma * (r[at - 1] + (r[at] - r[at - 1]) * (frac - c0) / (c1 - c0))
    p2 = (0.5 + q / rq.clamp(min=1e-300) * new).clamp(1e-9, 1.0 - 1e-9)
    pos = torch.cat([p1, p2], 1).contiguous()
    d2 = (pos - 0.5).square().sum(0)
    rho = 0.5 + 0.5 * torch.exp(-0.5 * d2 / sigma**2) / ((2 * math.pi) ** 1.5 * sigma**3)
    return dict(pos=pos, vel=0.1 * _normal(g, 3, size), u=0.5 + _uniform(g, size),
                gamma=5.0 / 3.0, pmass=1.0 / size, h=HFACT * (1.0 / size / rho) ** (1.0 / 3.0),
                alpha=1.0, cfl=0.3, box=((0.0,) * 3, (1.0,) * 3), periodic=True)


def _disc(size, g, r_in=0.1, r_out=1.0, hor=0.05, q=0.25, mass=1e-3):
    """Keplerian gas disc around a unit point mass: Sigma ~ 1/r, c_s = hor r^-q."""
    rm = 0.5 * (r_in + r_out)
    spans = (r_out - r_in, 2 * math.pi * rm, 5.0 * hor * rm ** (1.5 - q))
    scale = (size / (spans[0] * spans[1] * spans[2])) ** (1.0 / 3.0)
    n1, n2, n3 = (max(m, int(math.ceil(s * scale))) for m, s in zip((2, 4, 2), spans))
    while n1 * n2 * n3 < size:
        n3 += 1
    cells = torch.tensor([n1, n2, n3], device="cuda", dtype=torch.float64)[:, None]
    w = (_grid(n1, n2, n3) + 0.5) / cells
    w = w + 0.1 * _normal(g, *w.shape) / cells
    w = w[:, torch.argsort(_uniform(g, w.shape[1]))[:size]]
    r = r_in + w[0].clamp(0.0, 1.0) * spans[0]
    phi = 2 * math.pi * torch.remainder(w[1], 1.0)
    height = hor * r ** (-q) * r**1.5
    z = height * torch.special.ndtri(w[2].clamp(1e-4, 1.0 - 1e-4))
    vk = r ** (-0.5)
    pos = torch.stack([r * torch.cos(phi), r * torch.sin(phi), z])
    vel = torch.stack([-vk * torch.sin(phi), vk * torch.cos(phi), torch.zeros_like(r)])
    rho = (mass / (2 * math.pi * spans[0] * r) * torch.exp(-0.5 * (z / height) ** 2)
           / (math.sqrt(2 * math.pi) * height))
    lo, hi = pos.amin(1) - 1e-3, pos.amax(1) + 1e-3
    return dict(pos=pos, vel=vel, u=1.5 * (hor * pos.square().sum(0) ** (-0.5 * q)) ** 2,
                gamma=5.0 / 3.0, pmass=mass / size, lp07=(hor, q, 1.0), point_mass=1.0,
                h=HFACT * (mass / size / rho) ** (1.0 / 3.0), alpha=0.5, cfl=0.3,
                box=(tuple(lo.tolist()), tuple(hi.tolist())), periodic=False)


def _soundwave(size, g, amp=1e-4, gamma=1.0001):
    """size^3 particles on a cubic lattice carrying a travelling 1e-4 wave, with seeded 1e-4
    velocity and energy noise (isothermal-like gamma)."""
    pos = (_grid(size, size, size) + 0.5) / size
    pos[0] = torch.remainder(pos[0] + amp / (2 * math.pi) * torch.cos(2 * math.pi * pos[0]), 1.0)
    n = pos.shape[1]
    wave = amp * torch.sin(2 * math.pi * pos[0])
    vel = amp * _normal(g, 3, n)
    vel[0] += wave
    u = (1.0 + amp * _normal(g, n)) / (gamma * (gamma - 1.0))
    return dict(pos=pos, vel=vel, u=u, gamma=gamma, pmass=1.0 / n,
                h=HFACT * (1.0 / n / (1.0 + wave)) ** (1.0 / 3.0), alpha=0.1, cfl=0.3,
                box=((0.0,) * 3, (1.0,) * 3), periodic=True)


_SETUPS = dict(sedov=_sedov, homogeneous=_homogeneous, clustered=_clustered, disc=_disc,
               soundwave=_soundwave)


def _inputs(case, seed):
    if case["setup"] == "sedov":
        return _sedov(case["size"], _gen(seed), case.get("jitter", 0.05))
    return _SETUPS[case["setup"]](case["size"], _gen(seed))


def _model(s, precision):
    m = sg.get_Model_SPH(context=sg.Context(), vector_type="f64_3", sph_kernel="M4")
    cfg = m.gen_default_config()
    if s.get("av") == "cd10":
        cfg.set_artif_viscosity_VaryingCD10(alpha_min=0.0, alpha_max=1.0, sigma_decay=0.1,
                                            alpha_u=1.0, beta_AV=2.0)
    else:
        cfg.set_artif_viscosity_Constant(alpha_u=1.0, alpha_AV=s["alpha"], beta_AV=2.0)
    if s["periodic"]:
        cfg.set_boundary_periodic()
    else:
        cfg.set_boundary_free()
    if "lp07" in s:
        cfg.set_eos_locally_isothermalLP07(*s["lp07"])
        cfg.add_ext_force_point_mass(s["point_mass"], 0.0)
        cfg.set_constant_G(1.0)
    else:
        cfg.set_eos_adiabatic(s["gamma"])
    cfg.set_particle_mass(s["pmass"])
    cfg.set_precision(precision)
    cfg.set_cfl_cour(s["cfl"])
    cfg.set_cfl_force(s["cfl"])
    m.set_solver_config(cfg)
    m.resize_simulation_box(*s["box"])
    n = s["pos"].shape[1]
    m.set_particles(torch.zeros(n, 3, dtype=torch.float64).numpy())
    for field, value in (("xyz", s["pos"]), ("vxyz", s["vel"]), ("hpart", s["h"]),
                         ("uint", s["u"])):
        m.get_field_tensor(field).copy_(value)
    return m


# ------------------------------------------------------------------------ passes
def prepare(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "modules":
        s["ctx"] = L.Context(0)
        s["precision"] = case["precision"]
        # the host solver's own neighbour list, 160 slots per particle
        s["list"] = torch.zeros(160 * s["h"].shape[0], dtype=torch.int32, device="cuda")
        return dict(kind="modules", s=s)
    m = _model(s, case["precision"])
    if case["kind"] == "step":
        return dict(kind="step", model=m, dt_zero=s.get("dt_zero", False),
                    fields=FIELDS + (("alpha_AV", "soundspeed", "divv", "curlv", "dtdivv")
                                     if s.get("av") == "cd10" else ()))
    # a rollout starts from a state whose h, a and du are those of its positions
    m.evolve_once()
    start = {k: m.get_field_tensor(k).clone()
             for k in ("xyz", "vxyz", "axyz", "hpart", "uint", "duint")}
    target = s["vel"] + 1e-4 * _normal(_gen(seed + 1000003), *s["vel"].shape)
    return dict(kind="rollout", model=m, start=start, dt=m.get_dt(), alpha=s["alpha"],
                steps=case["steps"], target=target, kinetic=case["setup"] == "disc")


def _run_step(st):
    m = st["model"]
    if st["dt_zero"]:
        m.set_next_dt(0.0)
    m.evolve_once()
    out = {k: m.get_field_tensor(k) for k in st["fields"]}
    out["next_dt"] = m.get_dt()
    return out


def _run_rollout(st):
    m, start = st["model"], st["start"]
    for k in ("axyz", "hpart", "duint"):
        m.get_field_tensor(k).copy_(start[k])
    m.set_time(0.0)
    m.set_next_dt(st["dt"])
    m.set_cfl_multipler(1.0)
    v0 = start["vxyz"].clone().requires_grad_(True)
    u0 = start["uint"].clone().requires_grad_(True)
    alpha = torch.tensor(st["alpha"], dtype=torch.float64, requires_grad=True)
    x, v, u = adjoint.rollout(m, v0, u0, alpha, st["steps"], checkpoint_every=3,
                              x0=start["xyz"])
    if st["kinetic"]:
        loss = 0.5 * v.square().sum()
    else:
        loss = (v - st["target"]).square().sum()
    loss.backward()
    return dict(x=x.detach(), v=v.detach(), u=u.detach(), loss=loss.detach(), gv=v0.grad,
                gu=u0.grad, galpha=alpha.grad)


def _run_modules(st):
    s = st["s"]
    ctx, pos, h = s["ctx"], s["pos"], s["h"]
    n = h.shape[0]
    modules.Tree(ctx, pos, (0.0,) * 3, (1.0,) * 3, 3, h=h, htol=1.1)
    csr = modules.neighbour_cache(ctx, n, 1.1, s["precision"])
    s["list"][:csr["entries"].shape[0]] = csr["entries"]
    h_new, eps = h.clone(), torch.full_like(h, 100.0)
    modules.h_iterate(ctx, csr, pos, h, h_new, eps, s["pmass"], 1.1, 1.1, iters=50)
    om = modules.omega(ctx, csr, pos, h_new, s["pmass"])
    P, cs = modules.eos_adiabatic(ctx, h_new, s["u"], s["pmass"], s["gamma"])
    a, du, vsig = modules.derivs_constAV(ctx, csr, pos, s["vel"], h_new, om, s["u"], P, cs,
                                         s["pmass"], 1.0, 1.0, 2.0, precision=s["precision"])
    return dict(cnt=csr["cnt"], entries=s["list"], h=h_new, eps=eps, omega=om, P=P, cs=cs,
                a=a, du=du, vsig=vsig)


def run(state):
    return {"step": _run_step, "rollout": _run_rollout, "modules": _run_modules}[
        state["kind"]](state)


def _count(case):
    size = case["size"]
    return {"sedov": 4 * size**3, "soundwave": size**3}.get(case["setup"], size)


def work(case):
    """The state read and written once per step; per neighbour the density sums (25
    operations, two Newton evaluations and Omega) and the force terms (110)."""
    n = _count(case)
    cd10 = case["setup"] == "homogeneous"
    step_bytes = n * 8 * (12 + 13 + (9 if cd10 else 0))
    step_flops = n * NEIGHBOURS * (3 * 25 + 110 + (60 if cd10 else 0))
    if case["kind"] == "rollout":
        # forward steps, and a backward of twice a step's operations; states kept as the
        # backward's inputs, cotangents in and out
        return dict(bytes=case["steps"] * 2 * step_bytes, flops=case["steps"] * 3 * step_flops)
    if case["kind"] == "modules":
        # positions, velocities, h, u in; neighbour list and fields out
        pairs = n * NEIGHBOURS * 1.331
        return dict(bytes=n * 8 * (8 + 10) + 4 * pairs, flops=step_flops)
    return dict(bytes=step_bytes, flops=step_flops)


# ------------------------------------------------------------------------ 64-bit values
def _pairs(pos, reach, box):
    """All pairs (a, b), a included, with separation at most max(reach_a, reach_b); their
    separation vectors (minimum image in a periodic box of sides ``box``)."""
    n, r_all = pos.shape[1], float(reach.max())
    order = torch.argsort(pos[0])
    xs = pos[0][order].contiguous()
    ia, ib = [], []
    for c0 in range(0, n, 512):
        rows = order[c0:c0 + 512]
        lo, hi = float(xs[c0]) - r_all, float(xs[min(c0 + 511, n - 1)]) + r_all
        cols = [order[int(torch.searchsorted(xs, lo)):int(torch.searchsorted(xs, hi, right=True))]]
        if box is not None and hi - lo >= box[0]:
            cols = [order]
        elif box is not None:
            if lo < 0.0:
                cols.append(order[int(torch.searchsorted(xs, lo + box[0])):])
            if hi > box[0]:
                cols.append(order[:int(torch.searchsorted(xs, hi - box[0], right=True))])
        cols = torch.cat(cols)
        d2 = 0.0
        for ax in range(3):
            d = pos[ax][rows][:, None] - pos[ax][cols][None, :]
            if box is not None:
                d = d - box[ax] * torch.round(d / box[ax])
            d2 = d2 + d * d
        r, c = torch.nonzero(d2 <= torch.maximum(reach[rows][:, None], reach[cols][None, :]) ** 2,
                             as_tuple=True)
        ia.append(rows[r])
        ib.append(cols[c])
    ia, ib = torch.cat(ia), torch.cat(ib)
    d = pos[:, ia] - pos[:, ib]
    if box is not None:
        b = torch.tensor(box, device=pos.device, dtype=pos.dtype)[:, None]
        d = d - b * torch.round(d / b)
    return ia, ib, d, d.square().sum(0).sqrt()


def _f(q):
    return torch.where(q < 1, 0.25 * (2 - q) ** 3 - (1 - q) ** 3,
                       0.25 * (2 - q).clamp(min=0.0) ** 3)


def _df(q):
    return torch.where(q < 1, -3 * q + 2.25 * q * q,
                       torch.where(q < 2, -3 + 3 * q - 0.75 * q * q, torch.zeros_like(q)))


def _sum(n, ia, v):
    return torch.zeros(n, device=v.device, dtype=v.dtype).index_add_(0, ia, v)


def _density(n, ia, r, h, pmass):
    q = r / h[ia]
    rho = _sum(n, ia, pmass / math.pi * _f(q) / h[ia] ** 3)
    drho = _sum(n, ia, -pmass / math.pi * (3 * _f(q) + q * _df(q)) / h[ia] ** 4)
    return rho, drho


def _newton(n, ia, r, h0, pmass, tol):
    """h solving sum_b m W(r, h) = m (hfact / h)^3, each update within a factor of 1.1 and
    the whole within 1.1 of h0; eps the last relative update, -1 where the limit was hit."""
    h, eps = h0.clone(), torch.full_like(h0, 100.0)
    for _ in range(50):
        go = eps > tol
        if not bool(go.any()):
            break
        rho, drho = _density(n, ia, r, h, pmass)
        rho_h = pmass * (HFACT / h) ** 3
        new = h - (rho - rho_h) / (drho + 3 * rho_h / h)
        new = torch.minimum(torch.maximum(new, h / 1.1), h * 1.1)
        over = new >= h0 * 1.1
        e = torch.where(over, -torch.ones_like(h), (new - h).abs() / h0)
        new = torch.where(over, h0 * 1.1, new)
        h, eps = torch.where(go, new, h), torch.where(go, e, eps)
    return h, eps


def _forces(n, ia, ib, d, r, vel, u, h, om, P, cs, pmass, alpha):
    """Accelerations, du/dt and signal speeds of the constant viscosity (alpha_u 1, beta 2)."""
    rho = pmass * (HFACT / h) ** 3
    use = ((r <= 2 * h[ia]) | (r <= 2 * h[ib])) & (r > 0)
    ia, ib, d, r = ia[use], ib[use], d[:, use], r[use]
    e, v = d / r, vel[:, ia] - vel[:, ib]
    vr = (v * e).sum(0)
    Fa = _df(r / h[ia]) / (math.pi * h[ia] ** 4)
    Fb = _df(r / h[ib]) / (math.pi * h[ib] ** 4)
    ra, rb = rho[ia], rho[ib]
    qa = (-0.5 * ra * (alpha * cs[ia] + 2.0 * vr.abs()) * vr).clamp(min=0.0)
    qb = (-0.5 * rb * (alpha * cs[ib] + 2.0 * vr.abs()) * vr).clamp(min=0.0)
    ga = (P[ia] + qa) / (ra * ra * om[ia]) * Fa
    f = -pmass * (ga + (P[ib] + qb) / (rb * rb * om[ib]) * Fb)
    acc = torch.stack([_sum(n, ia, f * e[c]) for c in range(3)])
    vsig_u = ((P[ia] - P[ib]).abs() / (0.5 * (ra + rb))).sqrt()
    cond = 0.5 * vsig_u * (u[ia] - u[ib]) * (Fa / (ra * om[ia]) + Fb / (rb * om[ib]))
    du = _sum(n, ia, pmass * (ga * vr + cond))
    vsig = torch.zeros_like(h).index_reduce_(0, ia, cs[ia] + 2.0 * vr.abs(), "amax")
    # the particle itself is a pair at rest
    return acc, du, torch.maximum(vsig, cs)


def exact(case, seed):
    """Plain torch in 64 bits for the first pass (dt = 0) of the adiabatic, constant-viscosity
    cases up to 300,000 particles: x, v and u stay, h solves the density constraint."""
    n = _count(case)
    if case["kind"] == "rollout" or case["setup"] in ("homogeneous", "disc") or n > 300000:
        return None
    if case["kind"] == "step" and case["setup"] == "clustered":
        return None  # some h leave the first neighbour search's reach
    s = _inputs(case, seed)
    module = case["kind"] == "modules"
    pmass, h0 = s["pmass"], s["h"]
    ia, ib, d, r = _pairs(s["pos"], 2.2 * h0, None if module else s["box"][1])
    h, eps = _newton(n, ia, r, h0, pmass, 1e-6 if module else 1e-13)
    _, drho = _density(n, ia, r, h, pmass)
    rho = pmass * (HFACT / h) ** 3
    om = 1 + h / (3 * rho) * drho
    P = (s["gamma"] - 1) * rho * s["u"]
    cs = (s["gamma"] * P / rho).sqrt()
    a, du, vsig = _forces(n, ia, ib, d, r, s["vel"], s["u"], h, om, P, cs, pmass, s["alpha"])
    if module:
        return dict(cnt=None, entries=None, h=h, eps=None, omega=om, P=P, cs=cs, a=a, du=du,
                    vsig=vsig)
    return dict(xyz=s["pos"], vxyz=s["vel"], axyz=a, hpart=h, uint=s["u"], duint=du, omega=om,
                next_dt=None)

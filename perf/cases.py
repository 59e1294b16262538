"""The work a user of this framework has it do, as cases to be timed.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (inputs on the GPU from a seed, and the geometry, solved once per
process like in a user's program), `run` is one pass through the public entry
points, `work` what the pass cannot do without, `exact` the same results in
plain 64-bit torch where they are computed numbers.

Ranges: geometries from the default hemisphere (39 panels) over the
2000-panel hemisphere-on-post to the 3000-panel cylindrical well; single
points and single electrons to some 10^5 points; groups of 1 to 256
electrons; both far-field rules (the reference quadrature is the default of
every entry point, the adaptive rule the one whole benchmark traces take).
Traces are kept to workloads whose endpoints are well conditioned: dense
bunches near a tip magnify a last-digit change to 1e-6 of the endpoint, which
says nothing about the code.
"""

import functools
import math

import numpy as np
import torch

from bem_b200 import engine, workloads
from bem_b200 import geometry as bg
from bem_b200.constants import COULOMB_CONSTANT, ELEMENTARY_CHARGE, SPEED_OF_LIGHT, ev_to_kg
from bem_b200.tracker import SpecificParticleTracer

DEV = "cuda"
F64 = torch.float64
MASS = ev_to_kg(workloads.ELECTRON_MC2_EV)
CM = -ELEMENTARY_CHARGE / MASS
PLUMMER = 1e-12
Z0 = 3e-9
R_POST, L_POST = 50e-9, 5e-6
R_WELL, H_WELL = 2e-6, 1e-6
R_BALL = 1e-6


def listed():
    return [
        # one line scan on the axis side of the tip, or one group's positions: latency
        dict(name="field_line", op="field", geo="post", rule="adaptive", n=33),
        # the field of the default hemisphere at a plot's points, every argument at its default
        dict(name="field_ball", op="field", geo="ball", rule="reference", n=4000),
        # the reference quadrature on the benchmark tip (2000 panels, 64,000 rings)
        dict(name="field_quadrature", op="field", geo="post", rule="reference", n=1500),
        # a field map of the benchmark tip
        dict(name="field_map", op="field", geo="post", rule="adaptive", n=200_000),
        # a field map inside and above the 3000-panel well, an odd count
        dict(name="field_map_well", op="field", geo="well", rule="adaptive", n=100_003),
        # one stage of the benchmark workload: field, pair sums and images of 2048 groups of 32
        dict(name="stage_post", op="stage", geo="post", rule="adaptive", groups=2048, size=32),
        # one stage with every argument at its default, ragged group size, in the well
        dict(name="stage_well", op="stage", geo="well", rule="reference", groups=21, size=17),
        # one stage of large groups on the flat cathode: pair sums and plane images
        dict(name="stage_flat", op="stage", geo="flat", rule="reference", groups=300, size=256),
        # the BEM image-charge force of a batch of small groups
        dict(name="image_force", op="image", geo="image_tip", groups=256, size=4),
        # a whole trace of single electrons (no in-group force) from the benchmark tip
        dict(name="trace_singles", op="trace", geo="post", rule="adaptive", groups=16384, size=1, t_max=20e-12),
        # a whole trace of uneven groups from a micrometre hemisphere
        dict(name="trace_ball", op="trace", geo="ball_fine", rule="adaptive", groups=512, size=32, t_max=2e-12),
        # the driver class, defaults throughout, from host arrays to host arrays: flat cathode, screen at 100 um
        dict(name="tracker_flat", op="tracker", geo="flat", rule="reference", groups=16, size=64, t_max=5e-12),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["field", "field", "field", "stage", "stage", "image", "trace", "trace", "tracker"])
    if op == "field":
        if rng.random() < 0.6:
            return dict(op=op, geo=rng.choice(["post", "well", "ball_fine"]), rule="adaptive", n=_logint(rng, 1, 200_000))
        geo = rng.choice(["post", "well", "ball"])
        return dict(op=op, geo=geo, rule="reference", n=_logint(rng, 1, 40_000 if geo == "ball" else 1500))
    if op == "stage":
        size = _logint(rng, 1, 256)
        geo = rng.choice(["post", "well", "flat"])
        if geo == "flat":
            return dict(op=op, geo=geo, rule="reference", groups=_logint(rng, 1, 300), size=size)
        if rng.random() < 0.6:
            return dict(op=op, geo=geo, rule="adaptive", groups=max(1, _logint(rng, 1, 65536) // size), size=size)
        return dict(op=op, geo=geo, rule="reference", groups=max(1, _logint(rng, 1, 400) // size), size=size)
    if op == "image":
        return dict(op=op, geo=rng.choice(["image_tip", "image_well"]), groups=_logint(rng, 1, 256), size=rng.randint(1, 6))
    if op == "trace":
        if rng.random() < 0.5:
            return dict(op=op, geo="post", rule="adaptive", groups=_logint(rng, 16, 16384), size=1, t_max=rng.uniform(2e-12, 20e-12))
        return dict(op=op, geo="ball_fine", rule="adaptive", groups=_logint(rng, 8, 512), size=_logint(rng, 2, 32),
                    t_max=rng.uniform(1.2e-12, 2e-12))
    return dict(op=op, geo="flat", rule="reference", groups=rng.randint(2, 16), size=rng.randint(2, 64),
                t_max=rng.uniform(2e-12, 6e-12))


@functools.lru_cache(maxsize=None)
def _geometry(name):
    """A geometry as a program keeps it: meshed and solved once."""
    if name == "post":    # the benchmark tip: hemisphere of 50 nm on a 5 um post
        g = bg.PostTipBEMGeometry(-1e6, R_POST, L_POST, n_cap=100, n_wall=900, n_subdiv=8, z0=Z0)
    elif name == "well":  # the benchmark well, 3000 panels
        g = bg.CylindricalWellBEMGeometry(-2.5e6, R_WELL, H_WELL, n_segments=3000)
    elif name == "ball":  # the hemisphere with its default mesh
        g = bg.HemisphericalTipBEMGeometry(-1e7, R_BALL)
    elif name == "ball_fine":
        g = bg.HemisphericalTipBEMGeometry(-1e7, R_BALL, field_max_length=R_BALL * math.pi / 600)
    elif name == "image_tip":
        g = bg.HemisphericalTipBEMGeometry(-1e7, R_POST, z0=Z0)
    elif name == "image_well":
        g = bg.CylindricalWellBEMGeometry(-2.5e6, R_WELL, H_WELL, z0=Z0)
    else:
        g = bg.FlatCathode(-1e7, z0=Z0, kill_z_below=0.0)
    if g.is_bem:
        g.bem_tables(DEV)
    return g


def _uniform(gen, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=gen, device=DEV, dtype=F64)


def _points(geo, n, gen, lowest):
    """Points where the field is asked for: from `lowest` above the emitting
    surface to some micrometres, as many in each decade of the distance (an
    electron's time per decade of its flight)."""
    if geo == "flat":
        x, y = (10e-6 * torch.randn(n, generator=gen, device=DEV, dtype=F64) for _ in range(2))
        z = 10 ** _uniform(gen, n, math.log10(lowest), -5)
        return torch.stack([x, y, z], -1)
    d = 10 ** _uniform(gen, n, math.log10(lowest), -4.7)
    ph = _uniform(gen, n, 0.0, 2 * math.pi)
    if geo in ("well", "image_well"):
        r = 0.95 * R_WELL * torch.sqrt(_uniform(gen, n))
        return torch.stack([r * torch.cos(ph), r * torch.sin(ph), d - H_WELL], -1)
    R, base = {"post": (R_POST, L_POST), "image_tip": (R_POST, 0.0)}.get(geo, (R_BALL, 0.0))
    th = _uniform(gen, n, 0.0, 0.6)
    r = R + d
    return torch.stack([r * torch.sin(th) * torch.cos(ph), r * torch.sin(th) * torch.sin(ph),
                        base + r * torch.cos(th)], -1)


def _emission(case, seed):
    """Positions, velocities and birth times on the emitting surface."""
    G, E = case["groups"], case["size"]
    if case["geo"] == "flat":
        d = workloads.flat_c0(n_groups=G, n_emit=E, seed=seed, sigma_xy=50e-6)
    else:
        geo = _geometry(case["geo"])
        if case["geo"] == "post":
            d = workloads.tip_c1(geo.profile, geo.sigma, n_groups=G, n_emit=E, seed=seed, R=R_POST, L=L_POST)
        else:
            sizes = workloads.log_uniform_sizes(np.random.default_rng(G), G, 1, E)  # the same for every seed
            d = workloads.tip_c4(geo.profile, geo.sigma, seed=seed, R=R_BALL, L=0.0, sizes=sizes)
    return d


class _Particles:
    """The ParticleGroup attributes the driver reads."""

    def __init__(self, d):
        for k, v in d.items():
            setattr(self, k, v)
        self.mass = workloads.ELECTRON_MC2_EV
        self.species_charge = -ELEMENTARY_CHARGE
        self.species = "electron"

    def __len__(self):
        return len(self.x)


def prepare(case, seed):
    geo = _geometry(case["geo"])
    gen = torch.Generator(device=DEV).manual_seed(seed)
    op = case["op"]
    if op == "field":
        return dict(op=op, rule=case["rule"], tables=geo.bem_tables(DEV), points=_points(case["geo"], case["n"], gen, 1e-11))
    if op in ("stage", "image"):
        n = case["groups"] * case["size"]
        pos = _points(case["geo"], n, gen, 1e-10 if op == "stage" else 1e-9)
        active = (torch.rand(n, generator=gen, device=DEV) < (0.6 if op == "stage" else 0.95)).to(torch.uint8)
        q = torch.full((n,), -ELEMENTARY_CHARGE, device=DEV, dtype=F64)
        st = dict(op=op, geo=geo, pos=pos, active=active, charge=q)
        if op == "stage":
            return dict(st, mass=torch.full_like(q, MASS), sizes=[case["size"]] * case["groups"], rule=case["rule"])
        offsets = torch.arange(case["groups"] + 1, device=DEV, dtype=torch.int64) * case["size"]
        return dict(st, offsets=offsets, size=case["size"], solution=geo.image_solution(DEV), struct=geo.to_struct())
    d = _emission(case, seed)
    if op == "tracker":
        return dict(op=op, geo=geo, particles=_Particles({k: v for k, v in d.items() if k != "group_sizes"}),
                    n_emit=case["size"], t_max=case["t_max"])
    t = lambda v: torch.as_tensor(v, device=DEV, dtype=F64)
    pos = t(np.stack([d["x"], d["y"], d["z"]], -1))
    vel = t(np.stack([d["px"], d["py"], d["pz"]], -1) * (ELEMENTARY_CHARGE / SPEED_OF_LIGHT / MASS))
    n = len(pos)
    return dict(op=op, pos=pos, vel=vel, birth=t(d["t"]), charge=t(np.full(n, -ELEMENTARY_CHARGE)),
                mass=t(np.full(n, MASS)), sizes=d["group_sizes"], t_max=case["t_max"],
                tracer=engine.Tracer(geo, device=DEV, z_max=1e-3, far_rule=case["rule"]))


def run(state):
    op = state["op"]
    if op == "field":
        return engine.bem_field(state["tables"], state["points"], far_rule=state["rule"])
    if op == "stage":
        return engine.accel(state["geo"], state["pos"], state["active"], state["charge"], state["mass"],
                            state["sizes"], CM, PLUMMER, far_rule=state["rule"])
    if op == "image":
        return state["solution"].force(state["pos"], state["charge"], state["active"], state["offsets"],
                                       state["size"], geometry=state["struct"])
    if op == "tracker":
        tr = SpecificParticleTracer(state["particles"], state["n_emit"], state["geo"], screens=[1e-6, 1e-4],
                                    t_out=[0.5e-12, 1.5e-12], rtol=1e-8, t_max=state["t_max"], z_max=1e-3)
        tr.run()
        return tr.final_state
    b = engine.GroupBatch(state["pos"], state["vel"], state["birth"], state["charge"], state["mass"], state["sizes"])
    state["tracer"].run(b, state["t_max"], 1e-9, 1e-12, PLUMMER, CM)
    return dict(pos=b.positions(), vel=b.velocities(), t_death=b.t_death, t=b.t)


def work(case):
    op = case["op"]
    panels = {"post": 2000, "well": 3000, "ball": 39, "ball_fine": 600, "flat": 0}.get(case["geo"], 100)
    # a point's field: 64 FLOPs for each ring of the quadrature it is asked in, or one 32-term expansion
    per_point = 64.0 * 32 * panels if case.get("rule") == "reference" else (384.0 if panels else 4.0)
    if op == "field":
        return {"bytes": 48.0 * case["n"] + 256.0 * panels, "flops": per_point * case["n"]}
    n = case["groups"] * case["size"]
    images = {"post": 4, "flat": 2}.get(case["geo"], 1)
    pairs = 20.0 * n * case["size"] * images
    if op == "stage":
        return {"bytes": 72.0 * n + 256.0 * panels, "flops": 0.6 * (per_point * n + 0.6 * pairs)}
    if op == "image":
        # right-hand sides and reconstruction: 17 modes at 52 profile nodes and 816 quadrature points per electron
        return {"bytes": 64.0 * n, "flops": n * 17 * (52 + 816) * 10.0}
    if op == "trace" and case["geo"] != "post":
        n = int(n / max(1.0, math.log(case["size"])))  # sizes are log-uniform in 1..size
    # 70 attempts of seven stages for each birth
    return {"bytes": 180.0 * n, "flops": 70 * 7.0 * (per_point * n + pairs) * 0.5 * case["size"]}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch

GX4, GW4 = np.polynomial.legendre.leggauss(4)
GX8, GW8 = np.polynomial.legendre.leggauss(8)


def _ellip(p):
    """K(1 - p), E(1 - p) by the arithmetic-geometric mean."""
    a, b = torch.ones_like(p), torch.sqrt(p)
    s, w = 0.5 * (1.0 - p), 0.5
    for _ in range(10):
        c = 0.5 * (a - b)
        a, b = 0.5 * (a + b), torch.sqrt(a * b)
        w *= 2.0
        s = s + w * c * c
    K = 0.5 * math.pi / a
    return K, K * (1.0 - s)


def _ring(rho, z, a):
    """Field (E_rho, E_z) of unit-charge rings of radius a."""
    z2, a2, r2 = z * z, a * a, rho * rho
    D, d2 = (rho + a) ** 2 + z2, (rho - a) ** 2 + z2
    K, E = _ellip(d2 / D)
    sD = torch.sqrt(D)
    er = (K - (a2 - r2 + z2) * E / d2) / (4 * math.pi**2 * rho * sD)
    ez = z * E / (2 * math.pi**2 * sD * d2)
    x2 = a2 + z2
    axis = r2 < 1e-10 * x2
    s = torch.sqrt(x2)
    er = torch.where(axis, rho * (2 * z2 - a2) / (8 * math.pi * x2 * x2 * s), er)
    ez = torch.where(axis, z / (4 * math.pi * x2 * s)
                     + 3 * r2 * z * (3 * a2 - 2 * z2) / (16 * math.pi * x2 * x2 * x2 * s), ez)
    return er, ez


def _exact_field(geo, pts):
    """Perturbation field at pts [n, 3]: on-surface offset, Gauss-4 on the
    sub-panels of far segments, sinh-mapped Gauss-8 on near ones."""
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=DEV, dtype=F64)
    prof, sig = t(geo.profile), t(geo.sigma)
    p0, tan = prof[:-1], prof[1:] - prof[:-1]
    L = torch.linalg.vector_norm(tan, dim=1)
    u = tan / L[:, None]
    nrm = torch.stack([-u[:, 1], u[:, 0]], 1)
    S, sub = len(L), geo.n_subdiv
    tq = t(((np.arange(sub)[:, None] + 0.5 * (GX4 + 1.0)) / sub).reshape(-1))
    wq = t(np.tile(0.5 * GW4 / sub, sub))
    rq, zq = (p0[:, k:k + 1] + tq * tan[:, k:k + 1] for k in (0, 1))
    dens = sig[:-1, None] + tq * (sig[1:] - sig[:-1])[:, None]
    w = 2 * math.pi * rq * L[:, None] * wq * dens
    gx, gw = t(GX8), t(GW8)
    out = []
    step = max(1, min(len(pts), 20_000_000 // (S * len(tq))))
    for c0 in range(0, len(pts), step):
        p = pts[c0:c0 + step]
        rho, z = torch.hypot(p[:, 0], p[:, 1]), p[:, 2]
        dr, dz = rho[:, None] - p0[:, 0], z[:, None] - p0[:, 1]
        al = torch.clamp((dr * tan[:, 0] + dz * tan[:, 1]) / (L * L), 0.0, 1.0)
        q2 = (dr - al * tan[:, 0]) ** 2 + (dz - al * tan[:, 1]) ** 2
        d2, s = torch.min(q2, dim=1)
        off = torch.where(d2 < (1e-9 * L[s]) ** 2, 1e-4 * L[s], torch.zeros_like(d2))
        re, ze = torch.where(rho == 0, rho, rho + off * nrm[s, 0]), z + off * nrm[s, 1]
        dr, dz = re[:, None] - p0[:, 0], ze[:, None] - p0[:, 1]
        proj = torch.minimum(torch.clamp(dr * u[:, 0] + dz * u[:, 1], min=0.0), L)
        dist = torch.sqrt((dr - proj * u[:, 0]) ** 2 + (dz - proj * u[:, 1]) ** 2)
        near = dist < L
        er, ez = _ring(re[:, None, None], ze[:, None, None] - zq, rq)
        far = torch.where(near, torch.zeros_like(dist), torch.ones_like(dist))[:, :, None] * w
        sr, sz = (far * er).sum((1, 2)), (far * ez).sum((1, 2))
        k, s = torch.nonzero(near, as_tuple=True)
        if len(k):
            pj, Ls = proj[k, s], L[s]
            d = torch.maximum(dist[k, s], 1e-15 * Ls)
            lo, hi = torch.asinh(-pj / d), torch.asinh((Ls - pj) / d)
            cnt = torch.clamp(torch.ceil((hi - lo) / 0.5), min=1.0)
            iv = torch.arange(int(cnt.max()), device=DEV, dtype=F64)
            width = ((hi - lo) / cnt)[:, None, None]
            v = lo[:, None, None] + (iv[None, :, None] + 0.5 * (gx + 1.0)) * width
            sl = pj[:, None, None] + d[:, None, None] * torch.sinh(v)
            a = p0[s, 0][:, None, None] + sl * u[s, 0][:, None, None]
            zz = p0[s, 1][:, None, None] + sl * u[s, 1][:, None, None]
            dn = sig[s][:, None, None] + sl / Ls[:, None, None] * (sig[s + 1] - sig[s])[:, None, None]
            er, ez = _ring(re[k][:, None, None], ze[k][:, None, None] - zz, a)
            ww = dn * 2 * math.pi * a * d[:, None, None] * torch.cosh(v) * 0.5 * width * gw
            ww = torch.where(iv[None, :, None] < cnt[:, None, None], ww, torch.zeros_like(ww))
            sr.index_add_(0, k, torch.nan_to_num(ww * er).sum((1, 2)))
            sz.index_add_(0, k, torch.nan_to_num(ww * ez).sum((1, 2)))
        safe = torch.where(rho > 0, rho, torch.ones_like(rho))
        out.append(torch.stack([sr * p[:, 0] / safe, sr * p[:, 1] / safe, sz], 1))
    return torch.cat(out)


def _pairs(tgt, src, q_t, q_s):
    """Softened Coulomb force [G, E, 3] of sources [G, E, 3] on targets."""
    d = tgt[:, :, None, :] - src[:, None, :, :]
    r2 = (d * d).sum(-1) + PLUMMER**2
    c = COULOMB_CONSTANT * q_t[:, :, None] * q_s[:, None, :] / (r2 * torch.sqrt(r2))
    return (c[..., None] * d).sum(2)


def _exact_stage(case, st):
    geo, act = st["geo"], st["active"].bool()
    pos = st["pos"]
    field = torch.zeros_like(pos)
    field[:, 2] = torch.where(pos[:, 2] >= 0, geo.E_gun, 0.0)
    if geo.is_bem:
        z = pos[:, 2]
        s = torch.clamp((geo.z_handoff - z) / (0.5 * geo.z_handoff), 0.0, 1.0)
        w = (s * s * (3 - 2 * s))[:, None]
        rho = torch.hypot(pos[:, 0], pos[:, 1])
        if case["geo"] == "post":
            rk = geo.R * (1 - 1e-6)
            inside = ((rho <= rk) & (z <= geo.L)) | (rho**2 + (z - geo.L) ** 2 <= rk * rk) | (z < 0)
        else:
            inside = torch.where(rho >= geo.R * (1 - 1e-6), z <= 0, z <= -geo.H * (1 + 1e-6))
        bem = torch.zeros_like(pos)
        want = act & ~inside
        bem[want] = _exact_field(geo, pos[want])
        bem[:, 2] += torch.where(inside, 0.0, geo.E_gun)
        field = w * bem + (1 - w) * field
    shape = (case["groups"], case["size"])
    q = torch.where(act, st["charge"], 0.0).reshape(shape)
    out = []
    for g0 in range(0, shape[0], 64):
        p, qq = pos.reshape(*shape, 3)[g0:g0 + 64], q[g0:g0 + 64]
        f = _pairs(p, p, qq, qq)
        if case["geo"] == "flat":
            m = p * torch.tensor([1.0, 1.0, -1.0], device=DEV, dtype=F64)
            m[..., 2] -= 2 * geo.z0
            f = f + _pairs(p, m, qq, -qq)
        elif case["geo"] == "post":
            loc = p.clone()
            loc[..., 2] -= geo.L
            a = geo.R - geo.z0
            d = torch.linalg.vector_norm(loc, dim=-1)
            ball = loc * (a * a / (d * d))[..., None]
            qb = -qq * (a / d)
            flip = torch.tensor([1.0, 1.0, -1.0], device=DEV, dtype=F64)
            down = torch.tensor([0.0, 0.0, -2 * (geo.L + geo.z0)], device=DEV, dtype=F64)
            f = f + _pairs(loc, ball, qq, qb) + _pairs(loc, loc * flip + down, qq, -qq)
            f = f + _pairs(loc, ball * flip + down, qq, -qb)
        out.append(f.reshape(-1, 3))
    acc = CM * field + torch.cat(out) / MASS
    return torch.where(act[:, None], acc, 0.0)


def exact(case, seed):
    if case["op"] == "field":
        return _exact_field(_geometry(case["geo"]), prepare(case, seed)["points"])
    if case["op"] == "stage":
        return _exact_stage(case, prepare(case, seed))
    return None  # the image force needs its solve, and traces their whole integration, restated

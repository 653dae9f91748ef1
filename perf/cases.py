"""Cases by which the speed of the framework is followed.

Each case is one stretch of a simulation as a user's program runs it through the public
entry points.  For a single scene (`kind` dam2, cavity, lid, pois, dam3): a restart state
goes up, `steps` steps run (density re-initialisations among them), and the whole state
comes back into the program's own arrays, which is what a run does between two outputs
(the scenes' output interval is 100 steps).  `batch` advances the scenes of a resident
batch and collects every scene's state; `solve` is the whole `solve(...)` call of a
script, with its set-up and tear-down.

The restart state is a developed flow: the scene's lattice with seeded particle disorder
and a swirl of up to a twentieth of the sound speed (a parabolic profile in the channel).
Results of the FP64 form are taken as they come; those of the FP32-compensated form, whose
pair sums are formed in 32 bits, are taken as 32-bit arrays, as a renderer or a training
set takes them.
"""
import math

import numpy as np
import torch

import ethersph_gb300 as sph
from ethersph_gb300 import _abi, batch, scenes

# launch shapes of the FP32-compensated form (lanes of continuity, lanes of momentum, -,
# threads of a block): the library's default; the neighbour list read by two lanes (the
# autotuner's pick on 2D scenes of 50k particles and the served batches' shape); the list
# read by one lane (its pick on large 3D scenes)
SHAPES = {
    "default": None,
    "list2": (-1, _abi.LANES_LIST + 2, -1, 128),
    "list1": (1, _abi.LANES_LIST + 1, -1, 64),
}


def listed():
    return [
        # the smallest call: a coarse dam break, where launches and latency count
        dict(name="dam2_fp64_800", kind="dam2", dx=0.05, form="fp64", shape="default", steps=100),
        # the plain FP64 form (the entry points' default) on the 5,000-particle dry dam break
        dict(name="dam2_fp64_5k", kind="dam2", dx=0.02, form="fp64", shape="default", steps=100),
        # an odd-sized lid-driven cavity: walls with a velocity and background pressure
        dict(name="lid_fp64_10k", kind="lid", n=101, form="fp64", shape="default", steps=100),
        # the 65,536-particle thermal cavity, plain FP64
        dict(name="cavity_fp64_65k", kind="cavity", n=256, form="fp64", shape="default", steps=60),
        # a 3D dam break of the served size range, plain FP64
        dict(name="dam3_fp64_52k", kind="dam3", dx=0.0126, column="served", form="fp64", shape="default", steps=30),
        # a script's whole solve(...) call on a small scene
        dict(name="solve_fp64_2k", kind="solve", dx=0.03, form="fp64", shape="default", steps=60),
        # the FP32-compensated form as solve(..., precision=1) runs it, on the dry dam break
        dict(name="dam2_fp32_5k", kind="dam2", dx=0.02, form="fp32", shape="default", steps=100),
        # a periodic channel of the served range
        dict(name="pois_fp32_15k", kind="pois", n=61, form="fp32", shape="list2", steps=100),
        # the thermal cavity at the shape the autotuner picks for it
        dict(name="cavity_fp32_65k", kind="cavity", n=256, form="fp32", shape="list2", steps=100),
        # a cavity of a million particles: the largest 2D scene
        dict(name="cavity_fp32_1m", kind="cavity", n=1024, form="fp32", shape="default", steps=60),
        # a 432,000-particle 3D dam break at the shape the autotuner picks for it
        dict(name="dam3_fp32_432k", kind="dam3", dx=0.01, column="full", form="fp32", shape="list1", steps=30),
        # a served batch of uneven dam breaks
        dict(name="batch_fp32_10", kind="batch", scenes=10, mix=1, form="fp32", shape="list2", steps=50),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: the sizes of the scenes the repository's tests,
    served streams and benchmark use, log-uniform."""
    kind = rng.choice(["dam2", "cavity", "lid", "pois", "dam3", "batch", "solve"])
    form = rng.choice(["fp64", "fp32"])
    shape = "default" if form == "fp64" or kind == "solve" else rng.choice(["default", "list2", "list1"])
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 10), mix=rng.randrange(10 ** 6), form="fp32", shape="list2",
                    steps=rng.randint(30, 50))
    c = dict(kind=kind, form=form, shape=shape, steps=rng.randint(30, 100))
    if kind == "dam2":
        c["dx"] = round(_log(rng, 0.007 if form == "fp64" else 0.004, 0.05), 5)
    elif kind == "solve":
        c["dx"] = round(_log(rng, 0.015, 0.05), 5)
    elif kind == "cavity":
        c["n"] = int(_log(rng, 24, 230 if form == "fp64" else 700))
        c["steps"] = min(c["steps"], 60)
    elif kind == "lid":
        c["n"] = int(_log(rng, 24, 200 if form == "fp64" else 500))
    elif kind == "pois":
        c["n"] = rng.randint(20, 80)
    else:
        c["dx"] = round(_log(rng, 0.0128, 0.04), 5)
        c["column"] = "served" if form == "fp64" else rng.choice(["served", "full"])
        c["steps"] = rng.randint(10, 30)
    return c


# ------------------------------------------------------------------ inputs
def _scene(case):
    k = case["kind"]
    if k in ("dam2", "solve"):
        return scenes.dam_break_2d(dx=case["dx"])
    if k == "cavity":
        return scenes.natural_convection_2d(n=case["n"])
    if k == "lid":
        return scenes.lid_driven_cavity_2d(n=case["n"], reinit=30)
    if k == "pois":
        return scenes.poiseuille_periodic_2d(n_across=case["n"], kernel="CubicSpline")
    if case["column"] == "served":
        return scenes.dam_break_3d(dx=case["dx"], tank=(1.6, 0.4, 0.8), column=(0.4, 0.4, 0.65))
    return scenes.dam_break_3d(dx=case["dx"])


def _develop(s, rng):
    """A developed flow on scene s: particle disorder, a swirl that vanishes at the edges
    of the fluid (a parabolic profile on a periodic scene), densities a little off rest."""
    f = s.fluid
    x = f.x_vec_
    dx = s.meta["dx"]
    if s.periodic_x:
        y = x[:, 1]
        f.v_vec_[:, 0] = 4.0 * s.meta["umax"] * y * (s.meta["H"] - y) / s.meta["H"] ** 2
        f.v_vec_ += rng.uniform(-0.02, 0.02, x.shape) * s.meta["umax"]
    else:
        lo, hi = x.min(axis=0) - dx / 2, x.max(axis=0) + dx / 2
        u = (x - lo) / (hi - lo)
        amp = 0.05 * s.model.c_0_ * rng.uniform(0.8, 1.2)
        sx, sy = np.sin(math.pi * u[:, 0]), np.sin(math.pi * u[:, 1])
        shade = np.sin(math.pi * u[:, 2]) if x.shape[1] == 3 else 1.0
        L = hi - lo
        f.v_vec_[:, 0] = amp * shade * sx ** 2 * np.sin(2 * math.pi * u[:, 1]) * L[0] / max(L[0], L[1])
        f.v_vec_[:, 1] = -amp * shade * sy ** 2 * np.sin(2 * math.pi * u[:, 0]) * L[1] / max(L[0], L[1])
    x += rng.uniform(-0.08, 0.08, x.shape) * dx
    if s.periodic_x:
        x[:, 0] %= s.meta["L"]
    f.rho_ *= 1.0 + 1e-4 * rng.uniform(-1.0, 1.0, len(f))
    if hasattr(f, "t_"):
        f.t_[:] = np.clip(1.0 - x[:, 0], 0.0, 1.0) + rng.uniform(-1e-3, 1e-3, len(f))
    return s


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 17])
    if case["kind"] == "batch":
        sizes = np.random.default_rng(case["mix"])  # the scenes' sizes belong to the case
        return [_develop(scenes.random_dam_break_2d(sizes), rng) for _ in range(case["scenes"])]
    return _develop(_scene(case), rng)


FIELDS = ("x_vec_", "v_vec_", "rho_", "p_", "c_")


def _out_arrays(s):
    n, d = s.fluid.x_vec_.shape
    out = {k: np.zeros((n, d)) for k in ("x", "v")}
    for k in ["rho", "p", "c", "mass", "gap"] + (["t", "kappa", "cp"] if hasattr(s.fluid, "t_") else []):
        out[k] = np.zeros(n)
    return out


def prepare(case, seed):
    s = _inputs(case, seed)
    prec = 0 if case["form"] == "fp64" else 1
    st = dict(case=case, scene=s)
    if case["kind"] == "batch":
        proto = s[0].params(precision=prec)
        need = [batch.footprint(q, prec) for q in s]
        b = batch.Batch(proto, sum(n[0] for n in need), sum(n[1] for n in need) + 1, sum(n[2] for n in need), len(s))
        b.set_launch_shape(*SHAPES[case["shape"]])
        st["batch"] = b
        st["ids"] = [b.add_scene(q, first_step=1, nsteps=10 ** 9) for q in s]
    elif case["kind"] == "solve":
        st["start"] = {k: getattr(s.fluid, k).copy() for k in FIELDS}
    else:
        sim = sph.Simulation(s.params(precision=prec), s.n_fluid, s.n_wall)
        for w in s.walls:
            sim.upload_walls(w)
        if SHAPES[case["shape"]]:
            sim.set_launch_shape(*SHAPES[case["shape"]])
        st["sim"] = sim
        st["out"] = _out_arrays(s)
    return st


def _given(case, d):
    if case["form"] == "fp64":
        return d
    return {k: torch.from_numpy(a).to(torch.float32) for k, a in d.items()}


def run(st):
    case, s = st["case"], st["scene"]
    if case["kind"] == "batch":
        b = st["batch"]
        b.step(case["steps"])
        b.synchronize()
        got = {}
        for q, sid in enumerate(st["ids"]):
            d = b.download(sid)
            got["scene%d" % q] = _given(case, {k: d[k] for k in ("x", "v", "rho", "p", "c")})
        return got
    if case["kind"] == "solve":
        for k, a in st["start"].items():
            getattr(s.fluid, k)[:] = a
        sph.solve(s.fluid, *s.walls, s.kernel, s.model, s.td, check=s.check, domain_lo=s.domain_lo,
                  domain_hi=s.domain_hi, nsteps=case["steps"], precision=0 if case["form"] == "fp64" else 1)
        return _given(case, dict(zip(("x", "v", "rho", "p", "c"), (getattr(s.fluid, k) for k in FIELDS))))
    sim = st["sim"]
    sim.upload_fluid(s.fluid)
    sim.step(1, case["steps"])
    d = sim.download(s.n_fluid, out=st["out"])
    return _given(case, {k: d[k] for k in ("x", "v", "rho", "p", "c") + (("t",) if "t" in d else ())})


# ------------------------------------------------------------------ work
def _size(case):
    """(fluid particles, neighbours of one) of a case."""
    if case["kind"] == "batch":
        sizes = np.random.default_rng(case["mix"])
        return sum(scenes.random_dam_break_2d(sizes).n_fluid for _ in range(case["scenes"])), 28
    if case["kind"] in ("dam2", "solve"):
        return round(2.0 / case["dx"]) * round(1.0 / case["dx"]), 28
    if case["kind"] in ("cavity", "lid"):
        return case["n"] ** 2, 28
    if case["kind"] == "pois":
        return 4 * case["n"] ** 2, 28
    a, b, c = (0.4, 0.4, 0.65) if case["column"] == "served" else (0.6, 0.6, 1.2)
    return round(a / case["dx"]) * round(b / case["dx"]) * round(c / case["dx"]), 112


def work(case):
    """Bytes: the restart state read and the final state written once (8 bytes a value).
    Flops: per step and neighbour the geometry, kernel and the terms of continuity and
    momentum (about 70, 95 with heat), 60 a particle for state and integration."""
    n, nbr = _size(case)
    d = 3 if case["kind"] == "dam3" else 2
    heat = case["kind"] == "cavity"
    values = 2 * (2 * d + 5 + (3 if heat else 0))
    return {"bytes": 8.0 * n * values, "flops": float(case["steps"]) * n * (nbr * (95 if heat else 70) + 60)}


# ------------------------------------------------------------------ in 64 bits
def _kernel(name, q, sigma, h):
    """W and dW/dr at q = r / h."""
    t = (2.0 - q).clamp(min=0.0)
    if name == "CubicSpline":
        inner = q < 1.0
        W = torch.where(inner, 3.0 * q * q * (q - 2.0) + 4.0, t ** 3) * (sigma / 4.0)
        return W, torch.where(inner, q * (3.0 * q - 4.0), -t * t) * (0.75 * sigma / h)
    if name == "WendlandC2":
        return sigma * t ** 4 * (1.0 + 2.0 * q) / 16.0, -0.625 * sigma / h * q * t ** 3
    return (sigma * t ** 6 * (35.0 * q * q + 36.0 * q + 12.0) / 768.0,
            -sigma / h * (35.0 / 96.0 * q * q + 7.0 / 48.0 * q) * t ** 5)


def _pairs(xi, xj, rc, period):
    """Directed pairs (i, j) with |xi_i - xj_j| <= rc, coincident ones left out."""
    dev, dim = xi.device, xi.shape[1]
    lo = torch.minimum(xi.min(0).values, xj.min(0).values) - 1.5 * rc
    hi = torch.maximum(xi.max(0).values, xj.max(0).values) + 1.5 * rc
    n = [int(v) + 1 for v in ((hi - lo) / rc).tolist()]
    edge = torch.full((dim,), rc, dtype=torch.float64, device=dev)
    if period:
        n[0] = int(period / rc)
        edge[0] = period / n[0]
        lo[0] = 0.0
    ci, cj = (((a - lo) / edge).floor().long() for a in (xi, xj))
    top = torch.tensor(n, device=dev) - 1
    ci, cj = torch.minimum(ci.clamp(min=0), top), torch.minimum(cj.clamp(min=0), top)
    stride = [1, n[0], n[0] * n[1]][:dim]
    key = sum(cj[:, a] * stride[a] for a in range(dim))
    key, order = torch.sort(key)
    cells = math.prod(n)
    start = torch.searchsorted(key, torch.arange(cells + 1, device=dev))
    out_i, out_j, out_r = [], [], []
    for o in range(3 ** dim):
        off = [o // 3 ** a % 3 - 1 for a in range(dim)]
        c = [ci[:, a] + off[a] for a in range(dim)]
        if period:
            c[0] = c[0] % n[0]
        ok = torch.ones(len(xi), dtype=torch.bool, device=dev)
        for a in range(dim):
            ok &= (c[a] >= 0) & (c[a] < n[a])
        k = sum(c[a].clamp(0, n[a] - 1) * stride[a] for a in range(dim))
        b, m = start[k], torch.where(ok, start[k + 1] - start[k], torch.zeros_like(k))
        i = torch.repeat_interleave(torch.arange(len(xi), device=dev), m)
        first = torch.cumsum(m, 0) - m
        j = order[b[i] + torch.arange(len(i), device=dev) - first[i]]
        r = xi[i] - xj[j]
        if period:
            r[:, 0] -= period * torch.round(r[:, 0] / period)
        d2 = (r * r).sum(1)
        keep = (d2 <= rc * rc) & (d2 > 0.0)
        out_i.append(i[keep])
        out_j.append(j[keep])
        out_r.append(r[keep])
    return torch.cat(out_i), torch.cat(out_j), torch.cat(out_r)


def _simulate(s, steps, dev):
    T = lambda a: torch.as_tensor(np.array(a, dtype=np.float64), device=dev)
    f, ker, mod, td = s.fluid, s.kernel, s.model, s.td
    x, v, rho, m = T(f.x_vec_), T(f.v_vec_), T(f.rho_), T(f.mass_)
    n, dim = x.shape
    heat = hasattr(f, "t_")
    if heat:
        temp, kap, cp = T(f.t_), T(f.kappa_), T(f.cp_)
    cat = lambda get: T(np.concatenate([get(w) for w in s.walls]))
    wx, wn, wg = cat(lambda w: w.x_vec_), cat(lambda w: w.normal_vec_), cat(lambda w: w.gap_)
    wv = cat(lambda w: getattr(w, "v_vec_", np.zeros(w.x_vec_.shape)))
    if heat:
        hot = cat(lambda w: np.full(len(w), 1.0 if hasattr(w, "t_") else 0.0))
        wt = cat(lambda w: getattr(w, "t_", np.zeros(len(w))))
        wk = cat(lambda w: getattr(w, "kappa_", np.zeros(len(w))))
    h, rc, name = ker.h_, ker.influence_radius_, ker.kind.__name__
    sigma = (10.0 / 7.0 if dim == 2 else 1.0) / math.pi / h ** dim if name == "CubicSpline" else \
        (7.0 / (4.0 * math.pi) if dim == 2 else 21.0 / (16.0 * math.pi)) / h ** dim if name == "WendlandC2" else \
        (9.0 / (4.0 * math.pi) if dim == 2 else 495.0 / (256.0 * math.pi)) / h ** dim
    W0 = float(_kernel(name, torch.zeros(1, dtype=torch.float64), sigma, h)[0])
    gap = float(f.gap_[0])
    Wg = float(_kernel(name, torch.tensor([gap / h], dtype=torch.float64), sigma, h)[0])
    g = T(mod.body_force_vec_)
    nu, hh, dt, p_bg = mod.nu_0_, 0.01 * h * h, td.dt_, mod.p_0_ / mod.rho_0_ ** 2
    pressed = s.solve != _abi.SOLVE_FLUID_WALL
    period = s.domain_hi[0] - s.domain_lo[0] if s.periodic_x else 0.0
    for step in range(1, steps + 1):
        i, j, r = _pairs(x, x, rc, period)
        d = r.norm(dim=1)
        W, dW = _kernel(name, d / h, sigma, h)
        grad = r * (dW / d)[:, None]
        vij = v[i] - v[j]
        rho = rho + dt * torch.zeros_like(rho).index_add_(0, i, m[j] * (vij * grad).sum(1))
        rr = rho / mod.rho_0_
        p = mod.b_ * (rr ** mod.gamma_ - 1.0) + mod.p_0_
        c = mod.c_0_ * torch.sqrt(rr ** (mod.gamma_ - 1))
        P = p / rho ** 2
        both = P[i] + P[j]
        both = both + both.abs() * 0.01 * W / Wg
        fv = 4.0 * nu * (rho[i] + rho[j]) * d * dW / (rho[i] + rho[j]) ** 2 / (d * d + hh)
        dv = torch.zeros_like(v).index_add_(0, i, m[j, None] * (fv[:, None] * vij - both[:, None] * grad))
        if heat:
            keq = 2.0 * kap[i] * kap[j] / (kap[i] + kap[j])
            q = 2.0 * keq * d * dW / rho[i] / rho[j] / (d * d + hh) * (temp[i] - temp[j])
            dT = torch.zeros_like(rho).index_add_(0, i, q * m[j] / cp[i])
        new_rho = rho
        if td.density_reinitialized_interval_ and step % td.density_reinitialized_interval_ == 0:
            sw = (W0 * m / rho).index_add(0, i, W * m[j] / rho[j])
            new_rho = (W0 * m).index_add(0, i, W * m[j]) / sw
        # walls
        i, w, r = _pairs(x, wx, rc, period)
        d = r.norm(dim=1)
        W, dW = _kernel(name, d / h, sigma, h)
        nw, vw = wn[w], v[i] - wv[w]
        vert = (vw * nw).sum(1)
        psi = (r * nw).sum(1).abs()
        along = torch.sqrt((d * d - psi * psi).clamp(min=0.0))
        q = psi / wg[w]
        push = (0.01 * c[i] ** 2 + torch.where(vert > 0.0, 0.0, 1.0) * c[i] * vert.abs()) / h * (1.0 - q).abs() / q.sqrt()
        push = push * ((1.0 + torch.cos(math.pi * along / wg[w])) / 2.0).abs()
        push = torch.where((q > 1.0) | (along > wg[w]), torch.zeros_like(push), push)
        acc = push[:, None] * nw
        if pressed:
            both = P[i] + p_bg
            both = both + both.abs() * 0.01 * W / Wg
            acc = acc - (m[i] * both * dW / d)[:, None] * r
        fv = 8.0 * nu * rho[i] * d * dW / (2.0 * rho[i]) ** 2 / (d * d + hh)
        acc = acc + (m[i] * fv)[:, None] * (vw - vert[:, None] * nw)
        dv = dv.index_add_(0, i, acc)
        if heat:
            q = (kap[i] + wk[w]) * d * dW / rho[i] / mod.rho_0_ / (d * d + hh) * (temp[i] - wt[w]) / mod.cp_
            dT = dT.index_add_(0, i, q * m[i] * hot[w])
            temp = temp + dt * dT
            body = -g * mod.beta_ * (temp - mod.t_0_)[:, None]
        else:
            body = g
        v = v + dt * body + dt * dv
        x = x + dt * v - dv * (dt * dt / 2.0)
        if period:
            x[:, 0] = x[:, 0] - period * (x[:, 0] >= period).double() + period * (x[:, 0] < 0.0).double()
        rho = new_rho
    out = dict(x=x, v=v, rho=rho, p=p, c=c)
    if heat:
        out["t"] = temp
    return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = _inputs(case, seed)
    if case["kind"] == "batch":
        return {"scene%d" % q: _simulate(a, case["steps"], dev) for q, a in enumerate(s)}
    return _simulate(s, case["steps"], dev)

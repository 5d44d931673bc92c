"""The framework's work as a user's program has it do, one case per path.

Each case is a dict: `kind` names the path, the other entries its sizes and
options.  `prepare` builds what such a program holds before the call (a model
drawn from the seed, a context with its tables), `run` is one pass through the
public entry points, and `exact` is the same result from numpy / torch in 64
bits where a direct evaluation is short enough.  The models are the shapes of
`galic_b200.synth`: the isotropic halo, the halo with an exponential disk and
the halo + disk + bulge composite, on response grids of level 5 to 7 and force
grids of 64^2 to 256^2.
"""
import math

import numpy as np
import torch

from galic_b200 import GALIC_FORM_FP32, GALIC_FORM_FP64, Context, forcegrid, jeans, particles, sampling, synth
from galic_b200.ensemble import Ensemble
from galic_b200.serving import Server

FORMS = {"fp64": GALIC_FORM_FP64, "fp32": GALIC_FORM_FP32}
TORBIT_FAC = 5.0  # integration time of an orbit in orbital periods
# particles of each component as fractions of the total (halo, disk, bulge)
SHARES = {"halo": (1.0,), "halo_disk": (5 / 6, 1 / 6), "composite": (0.75, 0.175, 0.075)}
# orbit-steps per orbit by response-grid level (measured means, halo + disk; they vary by some 20 % with the shape)
STEPS_PER_ORBIT = {5: 1000.0, 6: 2000.0, 7: 4000.0}
OPS_PER_STEP = 365.0  # floating-point operations of one orbit step with both deposits


def listed():
    return [
        # one call of the per-orbit drop-in, as a host program written against the original function makes it
        {"name": "one_orbit", "kind": "orbit", "shape": "halo_disk", "level": 7, "nbin": 256},
        # response pass of a plain spherical model: 1e5 particles, 64 x 64 response grid
        {"name": "response_fp64_halo", "kind": "response", "shape": "halo", "n": 100000, "level": 6, "nbin": 256,
         "form": "fp64"},
        # response pass of a halo + disk model on the finest grid, drop-in precision
        {"name": "response_fp64_halo_disk", "kind": "response", "shape": "halo_disk", "n": 1200000, "level": 7,
         "nbin": 256, "form": "fp64"},
        # the same in the throughput form
        {"name": "response_fp32_halo_disk", "kind": "response", "shape": "halo_disk", "n": 1200000, "level": 7,
         "nbin": 256, "form": "fp32"},
        # construction of a spherical model: the response pass and an iteration of 100 repetitions of 0.1 % + 1
        # of the particles each
        {"name": "construct_fp64_halo", "kind": "construct", "shape": "halo", "n": 100000, "level": 6, "nbin": 256,
         "form": "fp64", "per_rep": 101, "reps": 100, "window_mib": 4096},
        # construction of a three-component model on the finest grid in the throughput form
        {"name": "construct_fp32_composite", "kind": "construct", "shape": "composite", "n": 60000, "level": 7,
         "nbin": 256, "form": "fp32", "per_rep": 201, "reps": 16, "window_mib": 2048},
        # many small halos of uneven sizes advanced together
        {"name": "ensemble", "kind": "ensemble", "models": 12, "n_min": 10000, "n_max": 60000, "level": 6},
        # construction requests served concurrently
        {"name": "serve", "kind": "serve", "jobs": 6, "n_min": 10000, "n_max": 40000, "level": 6, "iterations": 1,
         "reps": 20, "workers": 4},
        # tree-filled force grid of a halo + disk model
        {"name": "force_grid", "kind": "fill", "shape": "halo_disk", "n": 1200000, "nbin": 256},
        # target maps (density, then energy) of a halo + disk model from Monte-Carlo samples of each component
        {"name": "targets", "kind": "targets", "shape": "halo_disk", "ntarget": 20000001, "level": 7, "nbin": 256},
        # Jeans tables of a halo + tilted disk
        {"name": "jeans", "kind": "jeans", "shape": "halo_disk", "nbin": 256},
        # initial particles of a halo + disk model
        {"name": "particles", "kind": "particles", "shape": "halo_disk", "n": 1200000, "nbin": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["orbit", "response", "response", "construct", "construct", "ensemble", "serve", "fill",
                       "targets", "jeans", "particles"])
    shape = rng.choice(["halo", "halo_disk", "composite"])
    level = rng.choice([5, 6, 7])
    nbin = rng.choice([64, 100, 128, 193, 256])
    if kind == "orbit":
        return {"kind": kind, "shape": shape, "level": level, "nbin": nbin}
    if kind == "response":
        return {"kind": kind, "shape": shape, "n": _log_int(rng, 2000, 1200000), "level": level, "nbin": nbin,
                "form": rng.choice(["fp64", "fp32"])}
    if kind == "construct":
        n = _log_int(rng, 5000, 100000)
        per = _log_int(rng, 11, 201)
        reps = max(2, min(_log_int(rng, 4, 100), n // per, (10100 if level < 7 else 3216) // per))
        return {"kind": kind, "shape": shape, "n": n, "level": level, "nbin": nbin, "form": rng.choice(["fp64", "fp32"]),
                "per_rep": per, "reps": reps, "window_mib": rng.choice([512, 1024, 2048])}
    if kind == "ensemble":
        return {"kind": kind, "models": rng.randint(2, 12), "n_min": 3000, "n_max": _log_int(rng, 10000, 60000),
                "level": rng.choice([5, 6])}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(2, 6), "n_min": 3000, "n_max": _log_int(rng, 5000, 40000),
                "level": rng.choice([5, 6]), "iterations": rng.randint(1, 2), "reps": rng.randint(2, 10),
                "workers": rng.randint(1, 4)}
    if kind == "fill":
        return {"kind": kind, "shape": shape, "n": _log_int(rng, 3000, 1200000), "nbin": nbin}
    if kind == "targets":
        return {"kind": kind, "shape": shape, "ntarget": _log_int(rng, 30000, 20000000), "level": level, "nbin": nbin}
    if kind == "jeans":
        return {"kind": kind, "shape": shape, "nbin": nbin}
    return {"kind": kind, "shape": shape, "n": _log_int(rng, 2000, 1200000), "nbin": nbin}


# ------------------------------------------------------------------ inputs


def _components(shape, n, seed):
    """The shape's components with the seed's halo scale and disk mass (within 10 % of the usual ones)."""
    counts = [max(int(n * w), 32) for w in SHARES[shape]]
    a, md = np.random.default_rng(seed).uniform(0.9, 1.1, 2) * (30.0, 5.0)
    C = synth.Component
    if shape == "halo":
        return [C("halo", 100.0, a, counts[0], tovs=0)]
    if shape == "halo_disk":
        return [C("halo", 100.0 - md, a, counts[0], tovs=0), C("disk", md, 3.5, counts[1], z0=0.7, tovs=3)]
    return [C("halo", 98.5 - md, a, counts[0], beta=0.2, tovs=1), C("disk", md, 3.5, counts[1], z0=0.7, tovs=3),
            C("bulge", 1.5, 1.0, counts[2], tovs=0)]


def _model(shape, n, level, nbin, seed):
    extent = {}
    if shape == "halo_disk":  # out to 20 disk scale lengths, as synth.config_halo_disk
        extent = {"outer_frac": (70.0 / (30.0 + 70.0)) ** 2, "inner_frac": 1e-7}
    return synth.build_model(_components(shape, n, seed), seed=seed, level=level, fg_nbin=nbin, torbit_fac=TORBIT_FAC,
                             **extent)


def _halos(case, count, seed):
    """Anisotropic halos as synth.config_ensemble draws them, their particle counts in geometric steps."""
    rng = np.random.default_rng(seed)
    n = np.geomspace(case["n_min"], case["n_max"], count).astype(int)
    return [synth.build_model([synth.Component("halo", 100.0, float(rng.uniform(10.0, 50.0)), int(k),
                                               beta=float(rng.uniform(-0.5, 0.5)), tovs=1)],
                              seed=seed + q, level=case["level"]) for q, k in enumerate(n)]


def _sample_params(m):
    comps = {c["kind"]: c for c in m.meta["components"]}
    h, d, b = comps["halo"], comps.get("disk"), comps.get("bulge")
    return sampling.sample_params(Rmax=m.meta["rmax"], Halo_A=h["scale"], Disk_Z0=d["z0"] if d else 0.0,
                                  Disk_H=d["scale"] if d else 0.0, Bulge_A=b["scale"] if b else 0.0,
                                  HaloBetaParameter=h["beta"])


def _jeans_params():
    return jeans.jeans_params(streaming=(0.0, 0.0, 0.8, 0.0), r_over_z=(0.0, 1.0, 1.0, 1.0))


def _types(m):
    return [t for t in (1, 2, 3) if m.params.NType[t] > 0]


def _dispersion_tables(m, seed):
    """Smooth Jeans tables of galactic magnitudes, per type: disp_r, dispz, dispphi, tilted vR2 and vz2."""
    N = m.params.FG_Nbin
    iR, iz = np.meshgrid(np.arange(N), np.arange(N))
    rng = np.random.default_rng(seed)
    return {t: [np.ascontiguousarray(rng.uniform(1e3, 4e4) * np.exp(-iR / 60.0 - iz / 40.0) + 50.0)
                for _ in range(5)] for t in _types(m)}


def _fill_inputs(case, seed):
    m = _model(case["shape"], 96, 5, case["nbin"], seed)
    comps = _components(case["shape"], case["n"], seed)
    pos, mass = synth.fill_sample(comps, [c.n for c in comps], m.meta["rmax"], seed=seed)
    p = m.params
    return forcegrid.fill_params(p.FG_Nbin, p.FG_Rmin, p.FG_Fac, p.G, 0.01 * comps[0].scale, 0.4, 4.0, 4), pos, mass


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        count = case["models"] if kind == "ensemble" else case["jobs"]
        models = _halos(case, count, seed)
        if kind == "serve":
            return {"case": case, "models": models, "seed": seed % 65521}
        ctxs = []
        for m in models:
            ctxs.append(Context(m.params))
            ctxs[-1].load_model(m)
        return {"case": case, "ctxs": ctxs, "ensemble": Ensemble(ctxs)}
    if kind == "fill":
        fp, pos, mass = _fill_inputs(case, seed)
        return {"case": case, "fp": fp, "pos": pos, "mass": mass}
    if kind == "orbit":
        m = _model(case["shape"], 200, case["level"], case["nbin"], seed)
    elif kind in ("targets", "jeans"):
        m = _model(case["shape"], 200, case.get("level", 5), case["nbin"], seed)
    elif kind == "particles":
        m = _model(case["shape"], 200, 5, case["nbin"], seed)
        for c in _components(case["shape"], case["n"], seed):  # the call draws this many; the model's own are replaced
            m.params.NType[synth.TYPE_OF[c.kind]] = c.n
    else:
        m = _model(case["shape"], case["n"], case["level"], case["nbin"], seed)
    ctx = Context(m.params)
    ctx.load_model(m)
    state = {"case": case, "ctx": ctx, "model": m, "types": _types(m), "seed": seed % 65521}
    if kind == "construct":
        perm = np.random.default_rng(seed).permutation(m.n)
        count = case["per_rep"] * case["reps"]
        state["lists"] = np.ascontiguousarray(np.resize(perm, count).reshape(case["reps"], case["per_rep"]),
                                              dtype=np.int32)
    elif kind == "targets":
        state["sp"] = _sample_params(m)
        state["tables"] = _dispersion_tables(m, seed)
        for t, tabs in state["tables"].items():
            sampling.set_dispersion(ctx, t, *tabs)
    elif kind in ("jeans", "particles"):
        state["sp"], state["jp"] = _sample_params(m), _jeans_params()
        if kind == "particles":
            jeans.calculate_dispfield(ctx, state["sp"], state["jp"])
    return state


# ------------------------------------------------------------------ one pass


def _responses(ctx, types):
    return {t: [ctx.response(t, g) for g in range(10)] for t in types}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        state["ensemble"].calc_all()
        parts = [c.particles() for c in state["ctxs"]]
        return {"fits": np.stack([c.fit() for c in state["ctxs"]]),
                "grids": np.stack([_responses(c, (1,))[1] for c in state["ctxs"]]),
                "particles": [np.concatenate(a) for a in zip(*parts)]}
    if kind == "serve":
        with Server(64 << 30, workers=case["workers"]) as srv:
            ids = [srv.submit(m, form=GALIC_FORM_FP32, max_iterations=case["iterations"],
                              reps_per_iteration=case["reps"], fraction_per_rep=0.001, converge_rel=0.0,
                              seed=state["seed"] + k, want_velocities=True) for k, m in enumerate(state["models"])]
            done = [srv.wait(i) for i in ids]
        return [{"fit": r["fit"], "vel": r["vel"], "status": r["status"], "orbit_steps": r["orbit_steps"]}
                for r in done]
    if kind == "fill":
        dpotdr, dpotdz, pot, _ = forcegrid.force_grid_fill(state["fp"], state["pos"], state["mass"])
        return {"dpotdr": dpotdr, "dpotdz": dpotdz, "pot": pot}
    ctx, m = state["ctx"], state["model"]
    if kind == "orbit":
        k = state["seed"] % m.n
        tall, orbits, *grids = ctx.produce_orbit_response_field_mod(m.pos[k], m.vel[k], m.mass[k], m.tint[k],
                                                                    m.ptype[k])
        return {"tall": tall, "orbits": orbits, "grids": grids}
    if kind == "response":
        ctx.calc_all_response_fields(FORMS[case["form"]])
        return {"fit": ctx.fit(), "grids": _responses(ctx, state["types"]), "particles": ctx.particles()}
    if kind == "construct":
        form = FORMS[case["form"]]
        ctx.set_particles(m.pos, m.vel, m.mass, m.tint, m.vesc, m.ptype, m.ptargets)
        ctx.calc_all_response_fields(form)
        fits = ctx.optimize_reps(state["lists"], state["seed"], 0, form, case["window_mib"] << 20, fits=True)
        return {"fits": fits, "grids": _responses(ctx, state["types"]), "particles": ctx.particles()}
    if kind == "targets":
        stream = sampling.Stream(42 + state["seed"])
        sampling.sample_density_targets(ctx, state["sp"], case["ntarget"], stream, renormalize=True)
        sampling.sample_energy_targets(ctx, state["sp"], case["ntarget"], stream)
        return {"stacks": {t: sampling.get_targets(ctx, t) for t in state["types"]}, "position": stream.position}
    if kind == "jeans":
        return jeans.calculate_dispfield(ctx, state["sp"], state["jp"])
    stream = sampling.Stream(42 + state["seed"])
    arrays, low = particles.initialize_particles(ctx, state["sp"], TORBIT_FAC, stream)
    return {"arrays": arrays, "low": low, "position": stream.position}


# ------------------------------------------------------------------ what a pass cannot do without


def work(case):
    kind = case["kind"]
    L = case.get("level", 5)
    N = case.get("nbin", 256)
    tables = 8.0 * (3 * N * N + 3 * 4 ** L)
    ngrid = 4 ** L
    types = len(SHARES[case["shape"]]) if "shape" in case else 1
    step_ops = OPS_PER_STEP * STEPS_PER_ORBIT[L]
    if kind == "orbit":
        return {"bytes": tables + 40.0 * ngrid, "flops": step_ops}
    if kind == "response":
        return {"bytes": 128.0 * case["n"] + tables + 80.0 * types * ngrid, "flops": step_ops * case["n"]}
    if kind == "construct":
        tries = case["per_rep"] * case["reps"]
        # response pass, the tries' old and trial orbits, and 14 stack differences of ~12 operations per try
        return {"bytes": 196.0 * case["n"] + tables + 80.0 * types * ngrid,
                "flops": step_ops * (case["n"] + 2 * tries) + 14 * 12.0 * 4 / 3 * ngrid * tries}
    if kind in ("ensemble", "serve"):
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        count = case["models"] if kind == "ensemble" else case["jobs"]
        tries = 0 if kind == "ensemble" else case["iterations"] * case["reps"] * (1 + 0.001 * mean)
        return {"bytes": count * (128.0 * mean + tables + 80.0 * ngrid),
                "flops": count * (step_ops * (mean + 2 * tries) + 14 * 12.0 * 4 / 3 * ngrid * tries)}
    if kind == "fill":
        # ~ 30 accepted items and 45 opening tests per probe for every factor e of the particle count
        probes = 8.0 * N * N
        return {"bytes": 32.0 * case["n"] + 24.0 * N * N,
                "flops": probes * math.log(max(case["n"], 3)) * (30 * 19.0 + 45 * 11.0)}
    if kind == "targets":
        # density and energy samples: ~ 60 operations each to place, 4 and 20 deposits
        return {"bytes": 8.0 * types * (6 * 4 / 3 * ngrid + 5 * N * N),
                "flops": types * case["ntarget"] * (2 * 60.0 + 4 * 2 + 20 * 3 + 60)}
    if kind == "jeans":
        # force and density (~ 60 operations) at the integrand points, the recurrences
        tilt = 0 if case["shape"] == "halo" else 1
        return {"bytes": 8.0 * N * N * (3 + 8 * types),
                "flops": 60.0 * N * N * (50 * types + 100 * tilt) + 12.0 * 100 * N * N * tilt}
    # ~ 80 draws per particle of the velocity rejection, ~ 30 operations each
    return {"bytes": 176.0 * case["n"] + 8.0 * 8 * N * N, "flops": 80 * 30.0 * case["n"]}


# ------------------------------------------------------------------ 64-bit results without the framework


def exact(case, seed):
    if case["kind"] == "orbit":
        return _exact_orbit(case, seed)
    if case["kind"] == "targets" and case["shape"] != "composite":  # the bulge redraws one draw at a time
        return _exact_targets(case, seed)
    if case["kind"] == "jeans":
        return _exact_jeans(case, seed)
    return None  # whole passes take minutes; the tree walk and the particle stream have no short form


def _exact_orbit(case, seed):
    """Kick-drift-kick integration with the response grids' bilinear deposits (mass, v_r^2, v_t^2, v_q^2, v_p^2)."""
    m = _model(case["shape"], 200, case["level"], case["nbin"], seed)
    p = m.params
    k = seed % 65521 % m.n
    N, Nb = p.FG_Nbin, 1 << p.DG_MaxLevel
    lfg, ldg = math.log(p.FG_Fac), math.log(p.DG_Fac)
    typ = int(m.ptype[k])
    dR, dz = m.dpotdr.tolist(), m.dpotdz.tolist()
    vs, cs = m.vstream[typ].tolist(), m.cellsize.tolist()
    grids = np.zeros((5, Nb * Nb))

    def bilinear(T, i, j, fi, fj, n):
        return (T[i * n + j] * (1 - fi) * (1 - fj) + T[i * n + j + 1] * (1 - fi) * fj +
                T[(i + 1) * n + j] * fi * (1 - fj) + T[(i + 1) * n + j + 1] * fi * fj)

    def cell(br, bz, n):
        out = []
        for b in (max(br, 0.0), max(bz, 0.0)):
            i = int(b)
            out.append((n - 2, 1.0) if i >= n - 1 else (i, b - i))
        return out

    def fields(x):
        R, z = math.hypot(x[0], x[1]), abs(x[2])
        jd, kd = math.log(R / p.FG_Rmin + 1) / lfg, math.log(z / p.FG_Rmin + 1) / lfg
        (j, fj), (i, fi) = cell(jd, kd, N)
        v = bilinear(vs, i, j, fi, fj, N)
        if jd < N - 1 and kd < N - 1:
            aR, az = bilinear(dR, i, j, fi, fj, N), bilinear(dz, i, j, fi, fj, N)
            a = [aR * x[0] / R, aR * x[1] / R, -az if x[2] < 0 else az]
        else:
            r = math.sqrt(R * R + z * z)
            f = p.M200 / p.Halo_Mass * p.G * p.Halo_Mass / ((r + 1e-6 * p.Halo_A) * (r + p.Halo_A) ** 2)
            a = [-f * c for c in x]
        c = cell(math.log(R / p.DG_Rmin + 1) / ldg - 0.5, math.log(z / p.DG_Rmin + 1) / ldg - 0.5, Nb)
        return a, v, c

    def moments(x, v, vstr):
        R2 = x[0] * x[0] + x[1] * x[1]
        vq = (v[1] * x[0] - v[0] * x[1]) / math.sqrt(R2)
        T = (x[0] * x[2], x[1] * x[2], -R2)
        vx, vt = sum(a * b for a, b in zip(v, x)), sum(a * b for a, b in zip(v, T))
        return (1.0, vx * vx / (R2 + x[2] * x[2]), vt * vt / sum(t * t for t in T), vq * vq, (vq - vstr) ** 2)

    def deposit(w, c, f):
        (j, fj), (i, fi) = c
        for di, wi in ((0, 1 - fi), (1, fi)):
            for dj, wj in ((0, 1 - fj), (1, fj)):
                at = (i + di) * Nb + j + dj
                for g in range(5):
                    grids[g, at] += w * wi * wj * f[g]

    x, v = [float(c) for c in m.pos[k]], [float(c) for c in m.vel[k]]
    span = float(m.tint[k])
    a, vstr, c = fields(x)
    f = moments(x, v, vstr)
    tall, orbits, last, before = 0.0, 0, False, 0.0
    while not last:
        (j, _), (i, _) = c
        dt = min(p.TimeStepFactorOrbit * p.V200 / math.sqrt(sum(q * q for q in a)),
                 p.TimeStepFactorCellCross * cs[i * Nb + j] / math.sqrt(sum(q * q for q in v)))
        if span < dt + tall:
            dt, last = span - tall, True
        deposit(0.5 * dt, c, f)
        v = [v[q] + 0.5 * dt * a[q] for q in range(3)]
        x = [x[q] + dt * v[q] for q in range(3)]
        a, vstr, c = fields(x)
        v = [v[q] + 0.5 * dt * a[q] for q in range(3)]
        f = moments(x, v, vstr)
        deposit(0.5 * dt, c, f)
        tall += dt
        rad = sum(s * t for s, t in zip(v, x))
        orbits += rad > 0 and before < 0
        before = rad
    grids *= float(m.mass[k]) / tall
    return {"tall": tall, "orbits": int(orbits), "grids": list(grids)}


def _uniforms(seed, first, count, dev):
    """Draws first .. first + count - 1 (both even) of the Philox4x32-10 stream (seed, 0, 0), as doubles in [0, 1)."""
    M32 = 0xFFFFFFFF
    k = torch.arange(first // 2, (first + count) // 2, dtype=torch.int64, device=dev)
    c = [k & M32, k >> 32, torch.zeros_like(k), torch.zeros_like(k)]
    k0, k1 = seed & M32, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & M32) ^ c[1] ^ k0, p1 & M32, ((p0 >> 32) & M32) ^ c[3] ^ k1, p0 & M32]
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    u = [(c[0] << 21) | (c[1] >> 11), (c[2] << 21) | (c[3] >> 11)]
    return torch.stack(u, 1).reshape(-1).to(torch.float64) * 2.0 ** -53


def _exact_targets(case, seed):
    m = _model(case["shape"], 200, case["level"], case["nbin"], seed)
    p, sp, tabs = m.params, _sample_params(m), _dispersion_tables(m, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    L, N, G, want = p.DG_MaxLevel, 1 << p.DG_MaxLevel, 4 ** p.DG_MaxLevel, case["ntarget"]
    Nf = p.FG_Nbin
    chunk = 6 << 20

    def points(t, d):
        if t == 1:
            r = sp.Halo_A * (d[0] + d[0].sqrt()) / (1 - d[0])
            cz = 2 * d[2] - 1
            s = r * torch.sqrt((1 - cz) * (1 + cz))
            R, phi, z = s, 2 * math.pi * d[1], r * cz
            ok = r <= sp.Rmax
        else:
            z = sp.Disk_Z0 / 2 * torch.log(d[0] / (1 - d[0]))
            R = torch.ones_like(z)
            live = torch.ones_like(z, dtype=torch.bool)
            while bool(live.any()):  # Newton steps until the radius moves by less than 1e-7 of itself
                e = torch.exp(-R)
                new = torch.where(live, R + ((1 + R) * e + d[1] - 1) / (R * e), R)
                live = live & ((new - R).abs() / new > 1e-7)
                R = new
            R = R * sp.Disk_H
            phi = 2 * math.pi * d[2]
            ok = R * R + z * z <= sp.Rmax ** 2
        return R, z, ok & ((R * torch.cos(phi)) ** 2 + z * z < sp.Rmax ** 2)

    def cells(R, z, rmin, lfac, n, shift):
        out = []
        for q in (R, z):
            b = (torch.log(q / rmin + 1) / lfac - shift).clamp(min=0.0)
            i = b.floor().clamp(max=n - 2)
            out += [i.to(torch.int64), (b - i).clamp(max=1.0)]
        return out

    stacks = {t: [None] * 6 for t in _types(m)}
    position = 0
    for energy in (False, True):
        for t in _types(m):
            comp = m.meta["components"][t - 1]
            T = [torch.as_tensor(a, device=dev).reshape(-1) for a in tabs[t]]
            V = torch.as_tensor(m.vstream[t], device=dev)
            acc = torch.zeros(5 if energy else 1, G, dtype=torch.float64, device=dev)
            left = want
            while left > 0:
                first = position - position % 2
                u = _uniforms(42 + seed % 65521, first, chunk + 2, dev)[position - first:][:chunk]
                R, z, keep = points(t, u.reshape(-1, 3).unbind(1))
                kept = torch.cumsum(keep, 0)
                if int(kept[-1]) >= left:
                    end = int(torch.searchsorted(kept, left))
                    keep[end + 1:] = False
                    position += 3 * (end + 1)
                else:
                    position += chunk
                left -= int(keep.sum())
                R, z = R[keep], z[keep].abs()
                j, fj, i, fi = cells(R, z, p.DG_Rmin, math.log(p.DG_Fac), N, 0.5)
                w = [(1 - fi) * (1 - fj), (1 - fi) * fj, fi * (1 - fj), fi * fj]
                at = [i * N + j, i * N + j + 1, (i + 1) * N + j, (i + 1) * N + j + 1]
                val = [torch.ones_like(R)]
                if energy and comp["tovs"] == 0:
                    r = torch.sqrt(R * R + z * z)
                    b, f, _, _ = cells(r, r, p.FG_Rmin, math.log(p.FG_Fac), Nf, 0.0)
                    val += [T[0][b] * (1 - f) + T[0][b + 1] * f] * 4
                elif energy:  # velocity structure 3
                    b, f, a, g = cells(R, z, p.FG_Rmin, math.log(p.FG_Fac), Nf, 0.0)

                    def at_cell(X):
                        return (X[a * Nf + b] * (1 - f) * (1 - g) + X[(a + 1) * Nf + b] * (1 - f) * g +
                                X[a * Nf + b + 1] * f * (1 - g) + X[(a + 1) * Nf + b + 1] * f * g)

                    phi2 = at_cell(T[2])
                    val += [at_cell(T[3]), at_cell(T[4]), phi2, phi2 + at_cell(V) ** 2]
                for q, x in enumerate(val):
                    for c in range(4):
                        acc[q] += torch.bincount(at[c], weights=w[c] * x, minlength=G)
            for q in range(acc.shape[0]):
                lev = [acc[q].reshape(N, N) * (p.MType[t] / want)]
                for _ in range(L):
                    s = lev[0]
                    lev.insert(0, s[0::2, 0::2] + s[1::2, 0::2] + s[0::2, 1::2] + s[1::2, 1::2])
                if not energy:
                    lev[-1] = lev[-1] * (p.MType[t] / lev[-1].sum())
                stacks[t][q + 1 if energy else 0] = torch.cat([s.reshape(-1) for s in lev]).cpu().numpy()
    return {"stacks": stacks, "position": position}


def _exact_jeans(case, seed):
    m = _model(case["shape"], 200, 5, case["nbin"], seed)
    p, sp, jp = m.params, _sample_params(m), _jeans_params()
    N = p.FG_Nbin
    lfg = math.log(p.FG_Fac)
    Rg = p.FG_Rmin * (p.FG_Fac ** np.arange(2 * N + 3, dtype=np.float64) - 1.0)
    TR, TZ = m.dpotdr.reshape(N, N), m.dpotdz.reshape(N, N)

    def accel(R, z):
        R, z = np.broadcast_arrays(np.asarray(R, dtype=np.float64), np.asarray(z, dtype=np.float64))
        jd, kd = np.log(R / p.FG_Rmin + 1) / lfg, np.log(z / p.FG_Rmin + 1) / lfg
        j, i = np.minimum(jd, N - 2).astype(int), np.minimum(kd, N - 2).astype(int)
        fj, fi = jd - j, kd - i
        out = [T[i, j] * (1 - fi) * (1 - fj) + T[i, j + 1] * (1 - fi) * fj + T[i + 1, j] * fi * (1 - fj) +
               T[i + 1, j + 1] * fi * fj for T in (TR, TZ)]
        r = np.sqrt(R * R + z * z)
        far = p.M200 / p.Halo_Mass * p.G * p.Halo_Mass / ((r + 1e-6 * p.Halo_A) * (r + p.Halo_A) ** 2)
        inside = (jd < N - 1) & (kd < N - 1)
        return np.where(inside, out[0], -far * R), np.where(inside, out[1], -far * z)

    def density(t, R, z):
        with np.errstate(over="ignore"):
            if t == 2:
                h, z0 = sp.Disk_H, sp.Disk_Z0
                rho = p.Disk_Mass / (4 * math.pi * h * h * z0) * np.exp(-R / h) * (
                    2 / (np.exp(z / z0) + np.exp(-z / z0))) ** 2
            else:
                a, mass, front = ((p.Halo_A, p.Halo_Mass, p.Halo_A) if t == 1 else
                                  (p.Bulge_A, p.Bulge_Mass, p.Bulge_Mass))  # the original's bulge prefactor
                r = np.sqrt(R * R + z * z)
                rho = mass / (2 * math.pi) * front / (r + 1e-6 * a) / (r + a) ** 3
        return np.where(np.abs(rho) < 1e-25, 0.0, rho)

    def over(a, b):
        return np.where(b > 0, a / np.where(b > 0, b, 1.0), 0.0)

    def tilt(f, R, z):
        """(h, h / R) of the tilted velocity ellipsoid."""
        axis = (R <= 1e-12 * z) | (R == 0)
        al = np.arctan(z / np.where(axis, 1.0, R))
        den = np.cos(al) ** 2 - f * np.sin(al) ** 2 + (1 + f) / 2 * np.sin(2 * al) * np.tan(2 * al)
        h = (f - 1) / 2 * np.tan(2 * al) / den
        return np.where(axis, 0.0, h), np.where(axis, (f - 1) / f, h * np.tan(al)) / z

    out = {}
    R2, Z2 = np.meshgrid(Rg[:N], Rg[:N])  # [iz, iR]
    for t in _types(m):
        tab = {w: np.zeros((N, N)) for w in ("disp_r", "dispz", "dispphi", "vstream", "tilted_vz2", "tilted_vR2",
                                             "tilted_vz2_prime", "tilted_vR2_prime")}
        beta = sp.HaloBetaParameter if t == 1 else 0.0
        dens = density(t, R2, Z2)
        y, rows = 0.0, []
        for i in range(N + 1):  # spherical: Heun steps inwards, 50 per interval
            r0, r1 = (Rg[N + 2], Rg[N]) if i == 0 else (Rg[N - i + 1], Rg[N - i])
            dr = (r1 - r0) / 50
            r = r0 + dr * np.arange(51)
            safe = np.where(r > 0, r, 1.0)
            a = (density(t, np.abs(r), 0.0) * accel(np.abs(r), 0.0)[0]).tolist()
            c = (2 * beta / safe).tolist()
            for s in range(50):
                k0 = a[s] - c[s] * y
                if r[s + 1] > abs(dr) and r[s] > abs(dr):
                    y += dr * 0.5 * (k0 + (a[s + 1] - c[s + 1] * (y + dr * k0)))
                elif r[s] > abs(dr):
                    y += dr * k0
            if i:
                rows.append(y)
        tab["disp_r"][0] = over(np.array(rows[::-1]), density(t, Rg[:N], 0.0))
        integ = np.zeros(N)
        for i in range(N + 1):  # axisymmetric: trapezoids towards the plane, 50 per interval
            z0, z1 = (Rg[N], Rg[2 * N]) if i == 0 else (Rg[N - i], Rg[N - i + 1])
            z = z0 + (z1 - z0) / 50 * np.arange(51)[:, None]
            f = -accel(Rg[None, :N], z)[1] * density(t, Rg[None, :N], z)
            integ = integ + (0.5 * (f[1:] + f[:-1]) * ((z1 - z0) / 50)).sum(0)
            if i:
                tab["dispz"][N - i] = over(integ, dens[N - i])
        j = np.arange(N)
        lo, hi = np.where(j > 1, j - 1, 1), np.where(j < N - 1, j + 1, j)
        lo[0], hi[0] = 1, 2
        dz, aR = tab["dispz"], accel(R2, Z2)[0]
        up, dn = dens[:, hi] * dz[:, hi], dens[:, lo] * dz[:, lo]
        both = (up > 0) & (dn > 0)
        dlog = np.where(both, np.log(np.where(both, up, 1.0) / np.where(both, dn, 1.0)) / np.log(Rg[hi] / Rg[lo]), 0.0)
        kpar = jp.StreamingVelocityParameter[t]

        def split(vphi2, vz2):
            vs = np.where((vphi2 > 0) & (vphi2 >= vz2), kpar * np.sqrt(np.maximum(vphi2 - vz2, 0.0)), 0.0)
            tab["dispphi"], tab["vstream"] = np.where(vphi2 > 0, vphi2 - vs * vs, 0.0), vs

        split(dz + R2 * -aR + dz * dlog, dz)
        if m.params.TypeOfVelocityStructure[t] == 3:
            f = jp.DispersionRoverZratio[t]
            q = np.zeros((N, N))
            R = Rg[:N]
            for k in range(N - 2, -1, -1):  # method of lines towards the plane, 100 substeps per row
                step = (Rg[k] - Rg[k + 1]) / 100
                z = Rg[k + 1] + step * np.arange(100)[:, None]
                h1, hor = tilt(f, R[None, :], z)
                nb = np.where(h1 > 0, np.where(j == N - 1, -1, j + 1), np.where(j == 0, 1, j - 1))
                to = np.maximum(nb, 0)
                h2 = tilt(f, R[to], z)[0]
                dR = np.where(nb >= 0, R[to] - R[None, :], 1.0)
                pz = -density(t, R[None, :], z) * accel(R[None, :], z)[1]
                row = q[k + 1]
                for s in range(100):
                    dq = np.where(nb[s] >= 0, (h2[s] * row[to[s]] - h1[s] * row) / dR[s] + row * hor[s], 0.0)
                    row = row + (-pz[s] - dq) * step
                q[k] = row
            vz2 = over(q, dens)
            axis = R2 == 0
            al = np.arctan(Z2 / np.where(axis, 1.0, R2))
            cc, ss, t2 = np.cos(al), np.sin(al), np.tan(2 * al)
            den = cc * cc - f * ss * ss + (1 + f) / 2 * np.sin(2 * al) * t2
            vrvz = vz2 * ((f - 1) / 2 * t2) / den
            vr2 = vz2 * (f * cc * cc - ss * ss + (1 + f) / 2 * np.sin(2 * al) * t2) / den
            tab["tilted_vz2"] = vz2
            tab["tilted_vR2"] = np.where(axis, vz2 / f, vr2)
            tab["tilted_vz2_prime"] = np.where(axis, vz2 / f, vr2 * ss * ss - 2 * vrvz * ss * cc + vz2 * cc * cc)
            tab["tilted_vR2_prime"] = np.where(axis, vz2, vr2 * cc * cc + 2 * vrvz * ss * cc + vz2 * ss * ss)
            lo, hi = np.maximum(j - 1, 0), np.minimum(j + 1, N - 1)
            with np.errstate(divide="ignore", invalid="ignore"):
                zz = np.where(Z2 > 0, Z2, 1.0)
                h = np.where(Z2 > 0, tilt(f, R2, zz)[0], 0.0)
                v = tab["tilted_vR2"]
                rho = np.where(dens > 0, dens, 1.0)
                vphi2 = (v + R2 / rho * (dens[:, hi] * v[:, hi] - dens[:, lo] * v[:, lo]) / (Rg[hi] - Rg[lo]) +
                         R2 * -aR + R2 / rho * (dens[:, hi] * h[:, hi] * vz2[:, hi] -
                                                dens[:, lo] * h[:, lo] * vz2[:, lo]) / (Rg[hi] - Rg[lo]))
            split(np.where(dens > 0, vphi2, 0.0), v)
        out[t] = tab
    return out

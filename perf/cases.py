"""The work a user of this framework has it do, as cases that can be timed and
compared: runs of the reference's 2D model, of the 3D FP64 forms and of the
mixed form, a batch of replicas, and the two stress solves that are called by
themselves. Every case goes through the package's public entry points
(api.Engine, api.Batch, stz_solve_noalloc), and a run case returns what a
driver program keeps: the events of the pass, the mean fields and counters and,
where such a program reads them back, whole fields.

Event fields returned: step, kind, site, mode (whole numbers), time, dt, q and
total_rate. The margin of an event is not: it is a difference of two nearly
equal cumulative sums, a diagnostic and not a result. total_rate sums the rates
of all 20 modes over the whole grid, so it sees every site of the stored field.

Runs end long before their end strain (raised out of reach), so that a pass is
the same work however often it is called.
"""
import ctypes as C
import math

import numpy as np
import torch

from metallic_glasses_gb300 import api, configs

# grid extents the engine takes (2^a 3^b)
_EXTENTS_2D = (32, 48, 64, 72, 96, 128, 144, 192, 216, 256, 288, 384, 432, 512)
_EXTENTS_3D = (12, 16, 18, 24, 32, 36, 48, 54, 64)
_EXTENTS_INCR = (16, 24, 32, 48, 64, 72, 96, 128)
_EXTENTS_MIXED = (16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 256)


def listed():
    return [
        # the reference's main drives one step at a time and looks at the state
        # after each (KMC(), bmg.c:139-178): the smallest call, all latency
        {"name": "ref2d_64_one_step", "kind": "step2d", "n1": 64, "n2": 64, "soft": 0.3},
        # a small study grid of the reference's 2D model on its shipped input
        # (the grid of the parity runs), stress and eigenstrain read back
        {"name": "ref2d_64_run", "kind": "run2d", "n1": 64, "n2": 64, "solver": "fft", "soft": 0.0, "mro": 0.0,
         "load": "tension", "steps": 60, "fields": "all"},
        # the reference's shipped grid and input, early in a run: most sites
        # have never transformed
        {"name": "ref2d_512_run", "kind": "run2d", "n1": 512, "n2": 512, "solver": "fft", "soft": 0.0, "mro": 0.0,
         "load": "tension", "steps": 50, "fields": "loaded"},
        # late in a run (every site softened), crystal-like sites, a grid that
        # is neither square nor a power of two, the incremental update
        {"name": "ref2d_288x432_soft_incr", "kind": "run2d", "n1": 288, "n2": 432, "solver": "incr", "soft": 1.0,
         "mro": 0.15, "load": "tension", "steps": 50, "fields": "loaded"},
        # 3D FP64 form with the reference's method (a re-solve per event)
        {"name": "fp64_64", "kind": "run3d", "n0": 64, "n1": 64, "n2": 64, "solver": "fft", "load": "shear",
         "events": 50, "fields": "loaded"},
        # 3D FP64 form with the incremental update, the largest grid it is run on
        {"name": "fp64_128_incr", "kind": "run3d", "n0": 128, "n1": 128, "n2": 128, "solver": "incr", "load": "shear",
         "events": 30, "fields": "loaded"},
        # mixed form: a small uneven grid (lines of 36 sites have no pass of their own)
        {"name": "mixed_24x48x36", "kind": "mixed", "n0": 24, "n1": 48, "n2": 36, "df": "normal", "load": "shear",
         "events": 500, "period": 1000, "fp64": 0, "fields": "all"},
        # mixed form at 128^3 with an FP64 re-solve every 1000 events: the headline study
        {"name": "mixed_128", "kind": "mixed", "n0": 128, "n1": 128, "n2": 128, "df": "normal", "load": "shear",
         "events": 1000, "period": 1000, "fp64": 1, "fields": "loaded"},
        # mixed form at 256^3 with correlated barriers: the largest study
        {"name": "mixed_256_correlated", "kind": "mixed", "n0": 256, "n1": 256, "n2": 256, "df": "correlated",
         "load": "shear", "events": 1000, "period": 1000, "fp64": 0, "fields": "none"},
        # independent replicas of uneven size, temperature and strain rate in one batch
        {"name": "batch_32", "kind": "batch", "count": 32, "n_a": 32, "n_b": 48, "n_c": 64, "n_d": 96, "events": 64},
        # the stress solve alone on a caller's own device tensors
        {"name": "solve_48x54x36", "kind": "solve", "dim": 3, "n0": 48, "n1": 54, "n2": 36},
        # spatially varying moduli: the reference's polarisation fixed point, then the stress read back
        {"name": "inhom_256", "kind": "inhom", "n1": 256, "n2": 256, "spread": 0.3},
    ]


def draw(rng):
    kind = rng.choice(("step2d", "run2d", "run2d", "run3d", "run3d", "mixed", "mixed", "batch", "solve", "inhom"))
    if kind == "step2d":
        return {"kind": kind, "n1": rng.choice(_EXTENTS_2D), "n2": rng.choice(_EXTENTS_2D),
                "soft": round(rng.uniform(0.0, 1.0), 2)}
    if kind == "run2d":
        return {"kind": kind, "n1": rng.choice(_EXTENTS_2D), "n2": rng.choice(_EXTENTS_2D),
                "solver": rng.choice(("fft", "incr")), "soft": rng.choice((0.0, round(rng.uniform(0.0, 1.0), 2))),
                "mro": rng.choice((0.0, 0.15)), "load": rng.choice(("tension", "compression")),
                "steps": rng.randint(10, 60), "fields": "loaded"}
    if kind == "run3d":
        solver = rng.choice(("fft", "incr"))
        ext = _EXTENTS_3D if solver == "fft" else _EXTENTS_INCR
        return {"kind": kind, "n0": rng.choice(ext), "n1": rng.choice(ext), "n2": rng.choice(ext), "solver": solver,
                "load": rng.choice(("shear", "stress", "tension")), "events": rng.randint(10, 30), "fields": "loaded"}
    if kind == "mixed":
        n = [rng.choice(_EXTENTS_MIXED) for _ in range(3)]
        return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "df": rng.choice(("normal", "correlated")),
                "load": rng.choice(("shear", "stress")), "events": rng.randint(100, 500),
                "period": rng.choice((100, 1000)), "fp64": rng.choice((0, 1)), "fields": "none"}
    if kind == "batch":
        s = [rng.choice((16, 24, 32, 48, 64, 96)) for _ in range(4)]
        return {"kind": kind, "count": rng.randint(2, 32), "n_a": s[0], "n_b": s[1], "n_c": s[2], "n_d": s[3],
                "events": rng.randint(16, 64)}
    if kind == "solve":
        if rng.random() < 0.5:
            return {"kind": kind, "dim": 2, "n0": 1, "n1": rng.choice(_EXTENTS_2D), "n2": rng.choice(_EXTENTS_2D)}
        return {"kind": kind, "dim": 3, "n0": rng.choice(_EXTENTS_3D), "n1": rng.choice(_EXTENTS_3D),
                "n2": rng.choice(_EXTENTS_3D)}
    return {"kind": kind, "n1": rng.choice(_EXTENTS_2D[:10]), "n2": rng.choice(_EXTENTS_2D[:10]),
            "spread": round(rng.uniform(0.05, 0.4), 2)}


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return np.random.default_rng(seed)


def _params_2d(case, seed):
    p = configs.ref2d(case["n1"], case["n2"], seed=seed % 100000 + 1, end="1e9", xfrac=case.get("mro", 0.0), xq0="1.8",
                      loading={"tension": api.LOAD_TENSION,
                               "compression": api.LOAD_COMPRESSION}[case.get("load", "tension")],
                      solver=api.SOLVER_KERNEL if case.get("solver") == "incr" else api.SOLVER_FFT)
    return p


def _soft_state(case, seed, N, cap):
    """Softening left by earlier transformations at a share of the sites: the
    increment of the last one, the permanent softening up to its cap, and the
    rest of the temporary one."""
    rng = _rng([seed, 2])
    hit = rng.random(N) < case["soft"]
    xx, xy = 0.07 * rng.standard_normal(N), 0.07 * rng.standard_normal(N)
    prev = np.where(hit, np.stack([xx, -xx, xy]), 0.0)
    perm = np.where(hit, np.minimum(cap, 13 * (2 * xx * xx + 2 * xy * xy)), 0.0)
    temp = np.where(hit, 39 * (2 * xx * xx + 2 * xy * xy), 0.0) * (rng.random(N) < 0.2)
    tlast = np.where(hit, -rng.uniform(1e-7, 1.0, N), -1.0)
    return prev, perm, temp, tlast


def _set_soft(eng, prev, perm, temp, tlast):
    for c in range(3):
        eng.set_field(api.FIELD_PREV_DEPS, c, prev[c])
    eng.set_field(api.FIELD_PERM_SOFT, 0, perm)
    eng.set_field(api.FIELD_TEMP_SOFT, 0, temp)
    eng.set_field(api.FIELD_TLAST, 0, tlast)


def _step_inputs(case, seed):
    """Barriers, modes, eigenstrain and mean strain of a 2D grid, all from the
    seed, with the model's own distributions."""
    rng = _rng([seed, 1])
    N = case["n1"] * case["n2"]
    Q0 = 2.0 + 0.25 * rng.standard_normal((20, N))
    a, b = 0.07 * rng.standard_normal((2, 20, N))
    deps = np.stack([a, -a, b], axis=1)
    exx, exy = 0.004 * rng.standard_normal((2, N)) * (rng.random(N) < 0.3)
    eps0 = np.stack([exx, -exx, exy])
    ebar = np.array([2e-3, -7e-4, 1e-3])
    return Q0, deps, eps0, ebar


def _inhom_inputs(case, seed):
    rng = _rng([seed, 3])
    N = case["n1"] * case["n2"]
    a, b = 0.07 * rng.standard_normal((2, N)) * (rng.random(N) < 0.125)
    eps0 = np.stack([a, -a, b])
    lam, mu = 1 + case["spread"] * rng.uniform(-1, 1, (2, N))
    return eps0, lam, mu, np.array([2.0e-3, -7.0e-4, 1.1e-3])


_E, _NU = 69.46, 0.365 * 2                    # the shipped input, as Init() takes it (init.c:26-27)
_MU2 = _E / (2 + 2 * _NU)
_LAM2 = _E * _NU / (1 - _NU * _NU)
_MU3, _LAM3 = 35.0, 2 * 35.0 * 0.35 / 0.3


def _params_3d(case, seed):
    n = (case["n0"], case["n1"], case["n2"])
    p = configs.shear64(seed % 100000, n[2], eng_end=1e9)
    p.n[0], p.n[1], p.n[2] = n
    if case["load"] == "stress":
        p.loading = api.LOAD_STRESS
        p.applied_stress[api.XY] = 1.0
        p.strain_rate = 0.0
    elif case["load"] == "tension":
        p.loading = api.LOAD_TENSION
    return p


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step2d", "run2d"):
        p = _params_2d(case, seed)
        eng = api.Engine(p)
        if kind == "step2d":
            Q0, deps, eps0, ebar = _step_inputs(case, seed)
            for m in range(20):
                eng.set_field(api.FIELD_DF, m, Q0[m])
                for c in range(3):
                    eng.set_field(api.FIELD_DEPS, 3 * m + c, deps[m, c])
            for c in range(3):
                eng.set_field(api.FIELD_EPS0, c, eps0[c])
        if case["soft"] > 0:
            _set_soft(eng, *_soft_state(case, seed, eng.N, p.perm_soft_cap))
        if kind == "step2d":
            eng.set_mean_strain(ebar)
            eng.solve()
        else:
            eng.run(max_steps=12)  # past the first, purely elastic steps
        return {"kind": kind, "case": case, "engine": eng, "seen": len(eng.events())}
    if kind == "run3d":
        p = _params_3d(case, seed)
        p.solver = api.SOLVER_KERNEL if case["solver"] == "incr" else api.SOLVER_FFT
        eng = api.Engine(p)
        eng.run(max_events=4)
        return {"kind": kind, "case": case, "engine": eng, "seen": len(eng.events())}
    if kind == "mixed":
        p = _params_3d(case, seed)
        if case["df"] == "correlated":
            p.df_kind = api.DF_CORRELATED
            p.q0_sd = 0.15
            p.q0_corr_len = 4.0
        p.precision = api.PREC_MIXED
        p.solver = api.SOLVER_KERNEL
        p.resolve_period = case["period"]
        p.resolve_fp64 = case["fp64"]
        eng = api.Engine(p)
        eng.run(max_events=16)
        return {"kind": kind, "case": case, "engine": eng, "seen": len(eng.events())}
    if kind == "batch":
        rng = _rng([seed, 4])
        ps = []
        for i in range(case["count"]):
            n = case[("n_a", "n_b", "n_c", "n_d")[i % 4]]
            p = configs.mixed128((seed + i) % 100000, n)
            p.strain_rate = 0.5 * 10 ** rng.uniform(-5, -2)
            p.end_strain = 1e9
            p.mode_seed_set, p.mode_seed = 1, 0
            p.temperature = rng.uniform(325.0, 585.0)
            ps.append(p)
        b = api.Batch(ps)
        b.run(4)
        return {"kind": kind, "case": case, "batch": b, "seen": [len(r.events()) for r in b.replicas]}
    if kind == "solve":
        g = torch.Generator(device="cuda").manual_seed(seed)
        nc = 3 if case["dim"] == 2 else 6
        N = case["n0"] * case["n1"] * case["n2"]
        eps = 0.05 * torch.randn(nc, N, generator=g, device="cuda", dtype=torch.float64)
        return {"kind": kind, "case": case, "lib": api.load_library(), "eps": eps, "sig": torch.empty_like(eps),
                "ebar": (C.c_double * nc)(*(_solve_ebar(nc)))}
    p = _params_2d(case, seed)
    eng = api.Engine(p)
    eps0, lam, mu, ebar = _inhom_inputs(case, seed)
    for c in range(3):
        eng.set_field(api.FIELD_EPS0, c, eps0[c])
    eng.set_field(api.FIELD_LAMBDA, 0, lam * p.lambda_)
    eng.set_field(api.FIELD_MU, 0, mu * p.mu)
    eng.set_mean_strain(ebar)
    return {"kind": kind, "case": case, "engine": eng}


def _solve_ebar(nc):
    return [1.5e-3 / (c + 1) for c in range(nc)]


# -------------------------------------------------------------------- runs
def _events_out(ev):
    return {k: np.ascontiguousarray(ev[k]) for k in ("step", "kind", "site", "mode", "time", "dt", "q", "total_rate")}


def _scalars_out(sc):
    return {"time": sc["time"], "eps_avg": np.array(sc["eps_avg"]), "stress": np.array(sc["stress"]),
            "eps0_avg": np.array(sc["eps0_avg"]), "step": sc["step"], "kstep": sc["kstep"], "astep": sc["astep"],
            "estep": sc["estep"]}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "solve":
        lib = state["lib"]
        st = lib.stz_solve_noalloc(case["dim"], case["n0"], case["n1"], case["n2"],
                                   _LAM2 if case["dim"] == 2 else _LAM3, _MU2 if case["dim"] == 2 else _MU3,
                                   state["eps"].data_ptr(), state["ebar"], state["sig"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        if st != api.OK:
            raise RuntimeError(lib.stz_last_error().decode())
        return {"sigma": state["sig"]}
    if kind == "batch":
        b = state["batch"]
        b.run(case["events"])
        evs, stress, kstep = [], [], []
        for i, r in enumerate(b.replicas):
            ev = r.events(first=state["seen"][i])
            state["seen"][i] += len(ev)
            evs.append(ev)
            sc = r.scalars()
            stress.append(sc["stress"])
            kstep.append(sc["kstep"])
        return {"events": _events_out(np.concatenate(evs)), "stress": np.array(stress), "kstep": np.array(kstep)}
    eng = state["engine"]
    if kind == "inhom":
        eng.solve()
        return {"sigma": np.stack([eng.field(api.FIELD_SIGMA, c) for c in range(3)])}
    if kind == "step2d":
        eng.run(max_steps=1)
    elif kind == "run2d":
        eng.run(max_steps=case["steps"])
    else:
        eng.run(max_events=case["events"])
    ev = eng.events(first=state["seen"])
    state["seen"] += len(ev)
    out = {"events": _events_out(ev), "scalars": _scalars_out(eng.scalars())}
    which = case.get("fields", "none")
    if which != "none":
        mixed = kind == "mixed"
        nc = 5 if mixed else eng.nc
        loaded = nc - 1 if eng.nc == 6 else 0
        comps = range(nc) if which == "all" else (loaded,)
        out["sigma"] = np.stack([eng.field(api.FIELD_SDEV if mixed else api.FIELD_SIGMA, c) for c in comps])
        if not mixed or which == "all":
            comps = range(eng.nc) if which == "all" else (5 if eng.nc == 6 else 0,)
            out["eps0"] = np.stack([eng.field(api.FIELD_EPS0, c) for c in comps])
    return out


# -------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    n0, n1, n2 = case.get("n0", 1), case.get("n1", 1), case.get("n2", 1)
    N = n0 * n1 * n2
    lg = math.log2(max(N, 2))

    def solve_flops(nc, N):
        # forward and inverse real transforms, the operator on half the spectrum
        return nc * 2 * 2.5 * N * lg + 90 * nc * N / 2

    if kind in ("step2d", "run2d"):
        steps = case.get("steps", 1)
        # barriers and modes (20 x 4), stress and eigenstrain read, stress
        # written, softening state read
        b = 8 * N * (20 * 4 + 3 * 3 + (6 if case["soft"] > 0 else 0))
        f = N * 20 * (7 + 20) + (3 * 3 * 2 * N if case.get("solver") == "incr" else solve_flops(3, N))
        return {"bytes": float(steps * b), "flops": float(steps * f)}
    if kind == "run3d":
        b = 8 * N * (6 + 1 + 6 + (0 if case["solver"] == "incr" else 6)) + (8 * N * 36 / 8 if case["solver"] == "incr" else 0)
        f = N * 20 * (13 + 20) + (36 * 2 * N if case["solver"] == "incr" else solve_flops(6, N))
        return {"bytes": float(case["events"] * b), "flops": float(case["events"] * f)}
    if kind == "mixed":
        # five stress coordinates read and written, the barrier, the folded response table
        b = N * (44 + 60 / 8)
        f = N * (50 + 20 * 12)
        return {"bytes": float(case["events"] * b), "flops": float(case["events"] * f)}
    if kind == "batch":
        s = sum(case[("n_a", "n_b", "n_c", "n_d")[i % 4]] ** 3 for i in range(case["count"]))
        return {"bytes": float(case["events"] * s * (44 + 60 / 8)), "flops": float(case["events"] * s * 290)}
    nc = 6 if case.get("dim") == 3 else 3
    reps = 8 if kind == "inhom" else 1  # the fixed point takes several homogeneous solves
    return {"bytes": float(8 * N * (2 * nc + (2 if kind == "inhom" else 0))), "flops": float(reps * solve_flops(nc, N))}


# ------------------------------------------------- the same values in 64 bits
def _hooke(nc, lam, mu, e):
    nd = 2 if nc == 3 else 3
    s = 2 * mu * e
    s[:nd] = s[:nd] + lam * e[:nd].sum(0)
    return s


def _green_stress(shape, lam, mu, eps, ebar):
    """C:(eps - eps*) of the periodic medium with mean strain ebar by complex
    FFTs; on Nyquist planes the average over the signs of the Nyquist
    components (all of them together in 2D)."""
    nc = eps.shape[0]
    E = torch.fft.fftn(eps.reshape((nc,) + shape).to(torch.complex128), dim=(1, 2, 3))
    f, ny = [], []
    for ax in (2, 1, 0):
        n = shape[ax]
        k = torch.arange(n, dtype=torch.float64)
        w = torch.where(2 * k < n, k, k - n) / n if n > 1 else torch.zeros(1, dtype=torch.float64)
        view = [1, 1, 1]
        view[ax] = n
        f.append(w.reshape(view).expand(shape))
        ny.append(((2 * k == n) & (n > 1)).reshape(view).expand(shape))
    norm = torch.sqrt(f[0] ** 2 + f[1] ** 2 + f[2] ** 2)
    norm[0, 0, 0] = 1.0
    tau = _hooke(nc, lam, mu, E.clone())
    at = {3: ((0, 0), (1, 1), (0, 1)), 6: ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))}[nc]
    t = {}
    for c, (a, b) in enumerate(at):
        t[a, b] = t[b, a] = tau[c]
    d = 2 if nc == 3 else 3
    alpha = (lam + mu) / (lam + 2 * mu)
    flips = (0, 7) if nc == 3 else range(8)
    tot = torch.zeros_like(E)
    for sg in flips:
        g = [torch.where(ny[a] & bool(sg >> a & 1), -f[a], f[a]) / norm for a in range(3)]
        F = [sum(t[a, b] * g[b] for b in range(d)) for a in range(d)]
        G = sum(g[a] * F[a] for a in range(d))
        e = torch.stack([(F[a] * g[b] + F[b] * g[a]) / (2 * mu) - (alpha / mu) * G * g[a] * g[b] for a, b in at]) - E
        tot += _hooke(nc, lam, mu, e)
    tot /= len(flips)
    N = shape[0] * shape[1] * shape[2]
    z = torch.as_tensor(ebar, dtype=torch.float64) * N - E[:, 0, 0, 0]
    tot[:, 0, 0, 0] = _hooke(nc, lam, mu, z.reshape(nc, 1)).reshape(nc)
    return torch.fft.ifftn(tot, dim=(1, 2, 3)).real.reshape(nc, N)


def _hooke_inv2(lam, mu, s):
    e = s / (2 * mu)
    e[:2] = e[:2] - lam / (2 * mu * (2 * lam + 2 * mu)) * (s[0] + s[1])
    return e


def _exact_step(case, seed):
    Q0, deps, eps0, ebar = _step_inputs(case, seed)
    N = case["n1"] * case["n2"]
    sig = _green_stress((1, case["n1"], case["n2"]), _LAM2, _MU2, torch.from_numpy(eps0), ebar).numpy()
    kT = 300.0 * 1.380658e-23 / 1.60217733e-19
    V0 = 0.7 * 0.7 * 1.0
    Q = Q0
    if case["soft"] > 0:
        prev, perm, temp, tlast = _soft_state(case, seed, N, -math.log(0.6))
        t_temp = 1 / (1e13 * math.exp(-0.37 / kT))
        soft = perm + temp * np.exp(tlast / t_temp)
        n2 = np.sqrt(prev[0] ** 2 + prev[1] ** 2 + 2 * prev[2] ** 2) + 1e-17
        n1 = np.sqrt(deps[:, 0] ** 2 + deps[:, 1] ** 2 + 2 * deps[:, 2] ** 2) + 1e-17
        dm = (prev[0] * deps[:, 0] + prev[1] * deps[:, 1] + 2 * prev[2] * deps[:, 2]) / n1 / n2
        Q = Q0 * np.exp(-((1 + dm) ** 2 / 4) * soft)
    W = (sig[0] * deps[:, 0] + sig[1] * deps[:, 1] + 2 * sig[2] * deps[:, 2]) * V0 * 1e-18 / 1.60217733e-19
    R = float((V0 * 1e13 * np.exp(-(Q - W / 2) / kT)).sum())
    none = dict.fromkeys(("step", "kind", "site", "mode", "time", "dt", "q"))
    return {"events": {**none, "total_rate": np.array([R])},
            "scalars": dict.fromkeys(("time", "eps_avg", "stress", "eps0_avg", "step", "kstep", "astep", "estep"))}


def _exact_inhom(case, seed):
    eps0, lam, mu, ebar = _inhom_inputs(case, seed)
    e0 = torch.from_numpy(eps0)
    lam_s, mu_s = torch.from_numpy(lam * _LAM2), torch.from_numpy(mu * _MU2)
    eb = torch.from_numpy(ebar).reshape(3, 1)
    nrm = float(torch.linalg.norm(eb))
    tau0 = _hooke(3, lam_s, mu_s, e0.clone())
    eff = _hooke_inv2(_LAM2, _MU2, tau0 + _hooke(3, _LAM2 - lam_s, _MU2 - mu_s, e0 + eb))
    for it in range(101):
        last = eff
        sig = _green_stress((1, case["n1"], case["n2"]), _LAM2, _MU2, last, ebar)
        tot = _hooke_inv2(_LAM2, _MU2, sig.clone()) + last
        eff = 0.5 * _hooke_inv2(_LAM2, _MU2, tau0 + _hooke(3, _LAM2 - lam_s, _MU2 - mu_s, tot)) + 0.5 * last
        change = float(torch.sqrt(((eff - last) ** 2).sum() / last.shape[1]))
        if change < 1e-3 * nrm:
            break
    return {"sigma": sig.numpy()}


def exact(case, seed):
    if case["kind"] == "solve":
        g = torch.Generator(device="cuda").manual_seed(seed)
        nc = 3 if case["dim"] == 2 else 6
        N = case["n0"] * case["n1"] * case["n2"]
        eps = 0.05 * torch.randn(nc, N, generator=g, device="cuda", dtype=torch.float64)
        dim2 = case["dim"] == 2
        return {"sigma": _green_stress((case["n0"], case["n1"], case["n2"]), _LAM2 if dim2 else _LAM3,
                                       _MU2 if dim2 else _MU3, eps.cpu(), _solve_ebar(nc))}
    if case["kind"] == "step2d":
        return _exact_step(case, seed)
    if case["kind"] == "inhom":
        return _exact_inhom(case, seed)
    return None

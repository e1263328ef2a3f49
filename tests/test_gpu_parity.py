"""GPU parity: the CUDA engine (through its C ABI) against the reference's own
fixtures and against the CPU oracle.

Bars: (site, mode) event sequences identical; clocks and fields within 1e-10
relative (the plain FP64 form); the mixed form's stress error against an FP64
re-solve of its own eigenstrain <= 1e-5.
"""
import numpy as np
import pytest

from conftest import golden
from metallic_glasses_gb300 import api, configs
from ref2d_cases import MATERIAL_CASES, MRO_CASES, MRO_SWITCH_CASES, SF_CASES, SWITCH_CASES, check_mro_state, params_for

pytestmark = pytest.mark.gpu

FIELD_RTOL = 1e-10


def rel_err(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


# ----------------------------------------------------------------- solver
@pytest.mark.parametrize("model,shape", [
    (api.MODEL_GLOBAL3D, (8, 8, 8)), (api.MODEL_GLOBAL3D, (12, 6, 16)), (api.MODEL_GLOBAL3D, (16, 24, 32)),
    (api.MODEL_GLOBAL3D, (48, 48, 48)), (api.MODEL_REF2D, (1, 64, 64)), (api.MODEL_REF2D, (1, 48, 96)),
    (api.MODEL_REF2D, (1, 512, 512)),
])
def test_fft_green_solve_matches_oracle(engine_lib, oracle_lib, model, shape):
    """The hand-written R2C/C2R solve with the fused Green's pass against the
    oracle's complex-FFT solve that keeps the real part, as the reference does."""
    if model == api.MODEL_REF2D:
        p = configs.ref2d(shape[1], shape[2])
    else:
        p = configs.shear64(seed=2)
        p.n[0], p.n[1], p.n[2] = shape
    eng = api.Engine(p)
    ora = oracle_lib.Model(p)
    rng = np.random.default_rng(11)
    nc = eng.nc
    N = eng.N
    for c in range(nc):
        v = rng.standard_normal(N) * 0.02
        eng.set_field(api.FIELD_EPS0, c, v)
        ora.set_field(api.FIELD_EPS0, c, v)
    eng.solve()
    ora.solve()
    for c in range(nc):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), ora.field(api.FIELD_SIGMA, c)) < 1e-11
    eng.close()


# ----------------------------------------------------- reference fixtures
def _shear_prefix_ok(eng, g):
    """SHEAR mode: after an avalanche the reference's mean-strain correction
    (evolution.c:92-97, first component masked in every mode) zeroes the mean
    shear stress, and its divergence test |Stress[2]| < 1e-17 (bmg.c:402)
    then compares rounding noise of the field average. Where the engine's
    noise falls below the bound first, it stops there with status 2; the
    events up to that step must still be the reference's."""
    sc = eng.scalars()
    if sc["stopped"] != 2:
        return False
    ev = eng.events()
    X = g["X"]
    tr = ev[ev["kind"] != api.EV_ELASTIC]
    k = len(tr)
    assert k <= len(X)
    assert np.array_equal(np.stack([tr["step"], tr["kind"], tr["site"], tr["mode"]], 1), X[:k])
    last = int(sc["step"])
    assert (X[:, 0] == last).any() and (X[X[:, 0] == last, 1] == 1).all(), "stop must follow an avalanche"
    return True


@pytest.mark.parametrize("case", ["ref2d_64_tension_s123", "ref2d_32_shear_s7", "ref2d_32_tension_nosoft_s5"] + MRO_CASES +
                         SF_CASES + SWITCH_CASES + MRO_SWITCH_CASES + MATERIAL_CASES)
def test_ref2d_event_sequence_matches_reference(engine_lib, case):
    g = golden(case)
    p = params_for(g)
    eng = api.Engine(p)
    hdr = g["hdr"]
    eng.run(max_steps=int(hdr[1]))
    if "shear" in case and _shear_prefix_ok(eng, g):
        return
    ev = eng.events()
    tr = ev[ev["kind"] != api.EV_ELASTIC]
    X = g["X"]
    assert len(tr) == len(X)
    for col, k in ((0, "step"), (1, "kind"), (2, "site"), (3, "mode")):
        assert np.array_equal(tr[k], X[:, col]), "first mismatch in %s at %s" % (
            k, np.nonzero(tr[k] != X[:, col])[0][:3])
    sc = eng.scalars()
    assert [sc["step"], sc["kstep"], sc["astep"], sc["estep"]] == [int(v) for v in hdr[1:]]
    S = g["S"]
    last_time = {}
    for e in ev:
        last_time[int(e["step"])] = e["time"]
    t = np.array([last_time[int(s)] for s in S[:, 0] if int(s) in last_time])
    assert len(t) == len(S)
    assert np.abs(t - S[:, 2]).max() <= FIELD_RTOL * np.abs(S[:, 2]).max()
    for c in range(3):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), g["sigma"][c]) < FIELD_RTOL
        assert rel_err(eng.field(api.FIELD_EPS0, c), g["eps0"][c]) < FIELD_RTOL
    assert rel_err(eng.field(api.FIELD_TLAST), g["tlast"]) < FIELD_RTOL
    assert rel_err(eng.field(api.FIELD_PERM_SOFT), g["perm_soft"]) < FIELD_RTOL
    assert rel_err(eng.field(api.FIELD_TEMP_SOFT), g["temp_soft"]) < FIELD_RTOL
    assert np.allclose(sc["eps_avg"][:3], g["sc"][1:4], rtol=FIELD_RTOL, atol=1e-14)
    assert np.allclose(sc["stress"][:3], g["sc"][4:7], rtol=1e-9, atol=1e-12)
    if case in MRO_CASES + MRO_SWITCH_CASES:
        # the map bit for bit; the modes through the host's cos/sin (glibc of
        # the machine that runs the engine, not the one that made the fixture)
        # and the device-drawn barriers to an ulp
        check_mro_state(eng, g, exact=False)
    eng.close()


@pytest.mark.parametrize("no_sf", [1, 0])
def test_mro_map_matches_oracle(engine_lib, oracle_lib, no_sf):
    """Crystal-like sites drawn at 15 % (seed 11, 32^2, softening on) with the
    NO_SF_XTAL_MRO switch as shipped and switched off: the engine takes the
    oracle's transformations for 1500 thermal events, fields within 1e-10. The
    oracle is pinned bit for bit to the reference built either way on the same
    input (fixtures ref2d_32_mro_s11 and ref2d_32_mro_xsfoff_s11)."""
    from oracle import pyoracle
    kw = dict(end="0.5", seed="11", xfrac="0.15", xq0="1.8")
    p = configs.ref2d(32, 32, **kw)
    p.no_sf_xtal_mro = no_sf
    q = configs.ref2d(32, 32, defaults=pyoracle.default_params, from_input=pyoracle.params_from_input, **kw)
    q.no_sf_xtal_mro = no_sf
    eng = api.Engine(p)
    ora = oracle_lib.Model(q)
    eng.run(max_events=1500)
    ora.run(max_events=1500)
    a, b = eng.events(), ora.events()
    a, b = a[a["kind"] != api.EV_ELASTIC], b[b["kind"] != api.EV_ELASTIC]
    assert len(a) == len(b)
    for k in ("step", "kind", "site", "mode"):
        bad = np.nonzero(a[k] != b[k])[0]
        assert bad.size == 0, "first mismatch in %s at %d" % (k, bad[0])
    mro = eng.field(api.FIELD_MRO, 0)
    assert (mro == 1).sum() > 100 and np.isin(a["site"], np.nonzero(mro)[0]).any()
    for c in range(3):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), ora.field(api.FIELD_SIGMA, c)) < FIELD_RTOL
    eng.close()


def test_ref2d_deterministic(engine_lib):
    p = configs.ref2d(32, 32)
    a, b = api.Engine(p), api.Engine(p)
    a.run(max_events=200)
    b.run(max_events=200)
    assert np.array_equal(a.events(), b.events())


# ------------------------------------------------------------- 3D vs oracle
@pytest.mark.parametrize("solver", [api.SOLVER_FFT, api.SOLVER_KERNEL])
@pytest.mark.parametrize("cfg,events", [("stress32", 400), ("shear16", 400)])
def test_global3d_plain_matches_oracle(engine_lib, oracle_lib, cfg, events, solver):
    """The FP64 forms against the oracle's full re-solve per event: the FFT
    re-solve (the reference's method) and the incremental update."""
    p = configs.stress32() if cfg == "stress32" else configs.shear64(seed=5, n=16)
    p.solver = solver
    eng = api.Engine(p)
    ora = oracle_lib.Model(p)
    eng.run(max_events=events)
    ora.run(max_events=events)
    a, b = eng.events(), ora.events()
    assert len(a) == len(b)
    for k in ("step", "kind", "site", "mode"):
        assert np.array_equal(a[k], b[k])
    assert np.abs(a["time"] - b["time"]).max() <= FIELD_RTOL * np.abs(b["time"]).max()
    for c in range(6):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), ora.field(api.FIELD_SIGMA, c)) < FIELD_RTOL
        assert rel_err(eng.field(api.FIELD_EPS0, c), ora.field(api.FIELD_EPS0, c)) < FIELD_RTOL
    assert rel_err(eng.field(api.FIELD_DF), ora.field(api.FIELD_DF)) < 1e-15


@pytest.mark.parametrize("solver", [api.SOLVER_FFT, api.SOLVER_KERNEL])
def test_first_10k_events_match_oracle_32(engine_lib, oracle_lib, solver):
    """The 32^3 stress-controlled configuration (1 GPa of shear, seed 0): the
    plain FP64 form takes the oracle's (step, kind, site, mode) sequence for the
    first 10^4 events, at its times, and ends with its stress and eigenstrain
    fields within 1e-10 of their size; with the FFT re-solve after every event
    (the reference's method) and with the incremental update."""
    p = configs.stress32()
    p.solver = solver
    eng = api.Engine(p)
    ora = oracle_lib.Model(p)
    eng.run(max_events=10000)
    ora.run(max_events=10000)
    a, b = eng.events(), ora.events()
    assert len(a) == len(b) and (a["kind"] == api.EV_THERMAL).sum() == 10000
    for k in ("step", "kind", "site", "mode"):
        bad = np.nonzero(a[k] != b[k])[0]
        assert bad.size == 0, "first mismatch in %s at %d" % (k, bad[0])
    assert np.abs(a["time"] - b["time"]).max() <= FIELD_RTOL * np.abs(b["time"]).max()
    for c in range(6):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), ora.field(api.FIELD_SIGMA, c)) < FIELD_RTOL
        assert rel_err(eng.field(api.FIELD_EPS0, c), ora.field(api.FIELD_EPS0, c)) < FIELD_RTOL
    eng.close()
    ora.close()


@pytest.mark.parametrize("model", ["shear32", "ref2d64"])
def test_fp64_incremental_form_matches_resolve_form(engine_lib, model):
    """The FP64 incremental form against the FFT re-solve after every event
    (the reference's method) over 2000 events: shear loading at 32^3, and the
    reference's 2D model at 64^2 on its shipped input (per-site modes re-drawn
    at each transformation, softening, prints and their re-solves). The same
    events at the same times, stress fields within 1e-12 of their size (FP64
    rounding of 2000 updates of the linear solve) and the same mean stress
    (C:(ebar - <eps*>) of the solve against the solved field's mean)."""
    out = []
    for solver in (api.SOLVER_FFT, api.SOLVER_KERNEL):
        p = configs.shear64(seed=3, n=32) if model == "shear32" else configs.ref2d(64, 64)
        p.solver = solver
        eng = api.Engine(p)
        eng.run(max_events=2000)
        nc = 6 if model == "shear32" else 3
        out.append((eng.events(), np.stack([eng.field(api.FIELD_SIGMA, c) for c in range(nc)]), eng.scalars()))
        eng.close()
    (a, fa, sa), (b, fb, sb) = out
    assert sa["status"] == sb["status"] == 0 and sa["kstep"] == sb["kstep"] == 2000
    for k in ("step", "kind", "site", "mode"):
        assert np.array_equal(a[k], b[k]), k
    assert np.abs(a["time"] - b["time"]).max() <= 1e-12 * np.abs(a["time"]).max()
    assert np.abs(fa - fb).max() <= 1e-12 * np.abs(fa).max()
    assert np.allclose(sa["stress"], sb["stress"], rtol=0, atol=1e-12 * np.abs(fa).max())


def test_ensemble_stress_strain_curves_agree():
    """Ensemble-mean stress-strain curves of the mixed form and the FP64 plain
    form (shear loading at 250 K to 3 % shear strain through the elastic rise,
    thermal yield and softening; 16^3, seeds 0..15, the same seeds in both
    forms) within 1 % of the plain curve's peak. The two forms' trajectories
    part after some events, so the difference of the means is mostly the
    sampling noise of 16 realisations per form."""
    from metallic_glasses_gb300 import timing
    out = timing.ensemble(16, 16)
    print("ensemble 16^3: %s" % {k: out[k] for k in ("rel_diff_max", "rel_diff_mean", "forms")})
    assert out["strain_xy_max"] > 0.029
    assert out["forms"]["plain"]["thermal_events"] > 1000
    assert out["rel_diff_max"] < 0.01, out["rel_diff_max"]


def test_ref2d_512_matches_oracle(engine_lib, oracle_lib):
    """The reference's 2D model at its own 512 x 512 grid on its shipped input
    (softening on): the engine takes the oracle's transformations (the oracle
    is pinned to the reference's code at this grid) for 30 thermal events,
    with the clock and fields within 1e-10."""
    p = configs.ref2d(512, 512)
    eng = api.Engine(p)
    ora = oracle_lib.Model(configs.ref2d(512, 512))
    eng.run(max_events=30)
    ora.run(max_events=30)
    a, b = eng.events(), ora.events()
    assert len(a) == len(b) and (a["kind"] == api.EV_THERMAL).sum() == 30
    for k in ("step", "kind", "site", "mode"):
        assert np.array_equal(a[k], b[k]), k
    assert np.abs(a["time"] - b["time"]).max() <= FIELD_RTOL * np.abs(b["time"]).max()
    for c in range(3):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), ora.field(api.FIELD_SIGMA, c)) < FIELD_RTOL
        assert rel_err(eng.field(api.FIELD_EPS0, c), ora.field(api.FIELD_EPS0, c)) < FIELD_RTOL
    eng.close()
    ora.close()


def test_correlated_barrier_field_matches_oracle(engine_lib, oracle_lib):
    p = configs.grf256(n=16)
    p.precision = api.PREC_FP64
    p.solver = api.SOLVER_FFT
    eng = api.Engine(p)
    ora = oracle_lib.Model(p)
    a, b = eng.field(api.FIELD_DF), ora.field(api.FIELD_DF)
    assert np.abs(a - b).max() < 1e-10
    assert abs(a.mean() - 1.2) < 0.05


# ------------------------------------------------------------- mixed form
def test_mixed_rates_select_like_plain_for_a_while(engine_lib):
    """FP32 rates against the FP64 plain form on the same seed: the same
    events until a near-tie of the FP32 rates flips one."""
    pm = configs.mixed128(n=16)
    pp = configs.plain128(n=16)
    m, q = api.Engine(pm), api.Engine(pp)
    m.run(max_events=20)
    q.run(max_events=20)
    a, b = m.events(), q.events()
    same = 0
    for x, y in zip(a, b):
        if x["site"] != y["site"] or x["mode"] != y["mode"]:
            break
        same += 1
    assert same >= 5
    assert np.allclose(a["time"][:same], b["time"][:same], rtol=1e-5)


def test_mixed_stress_error_within_bound(engine_lib):
    """Stress error of the FP32 incremental field against FP64 re-solves of
    the same eigenstrain every 1000 events: relative L2 and max norms of the
    deviatoric stress <= 1e-5."""
    p = configs.mixed128(n=32, resolve_period=1000)
    m = api.Engine(p)
    m.run(max_events=3000)
    sc = m.scalars()
    assert sc["kstep"] == 3000 and sc["n_resolves"] == 3
    assert 0 < sc["stress_err_rms_worst"] < 1e-5
    assert sc["stress_err_max_worst"] < 1e-5


def test_mixed_first_resolve_error_small(engine_lib):
    """One event after the start: the incremental update of one voxel's
    response against the FP64 re-solve of the same state."""
    p = configs.mixed128(n=24, resolve_period=1)
    m = api.Engine(p)
    m.run(max_events=3)
    sc = m.scalars()
    assert sc["kstep"] == 3 and sc["n_resolves"] == 3
    assert 0 < sc["stress_err_rms_worst"] < 1e-6
    assert sc["stress_err_max_worst"] < 1e-6


@pytest.mark.parametrize("n", [32, 24])
def test_mixed_pair_resolve_matches_fp64(engine_lib, n):
    """The mixed form's field solves in FP32 pairs (the default) against the
    same solves in FP64 (resolve_fp64 = 1): after the start solve and three
    periodic re-solves of an n^3 run the stored FP32 field agrees to within one
    FP32 rounding, the events are the same, and the measured stress errors of
    the incremental field agree to 1e-4 of their size (the pair transform
    carries about 48 bits; its error norms are summed in FP32 per warp). At
    24^3 the wave numbers' 1/n is not a binary fraction and the transforms
    take radix-3 passes."""
    out = {}
    for fp64 in (0, 1):
        p = configs.mixed128(n=n, resolve_period=100)
        p.resolve_fp64 = fp64
        e = api.Engine(p)
        e.run(max_events=300)
        sc = e.scalars()
        assert sc["kstep"] == 300 and sc["n_resolves"] == 3
        out[fp64] = (e.events(), sc, np.stack([e.field(api.FIELD_SDEV, k) for k in range(5)]))
        e.close()
    (ea, sa, fa), (eb, sb, fb) = out[0], out[1]
    for k in ("site", "mode"):
        assert np.array_equal(ea[k], eb[k]), k
    scale = np.abs(fb).max()
    assert np.abs(fa - fb).max() <= 2 ** -23 * scale
    for k in ("stress_err_rms_worst", "stress_err_max_worst"):
        assert abs(sa[k] - sb[k]) <= 1e-4 * sb[k] + 1e-13, k


def test_displacement_gradient_is_the_solved_strain_3d(engine_lib):
    """3D displacement field (no reference code exists in 3D): its spectral
    symmetric gradient equals the fluctuation of the total strain of the stress
    solve, C^-1:sigma + eps*, on every wave vector off the Nyquist planes (where
    the operator is the average of the sign choices)."""
    p = configs.plain128(n=16)
    e = api.Engine(p)
    e.run(max_events=40)
    u = e.displacement()
    sig = np.stack([e.field(api.FIELD_SIGMA, c) for c in range(6)])
    eps0 = np.stack([e.field(api.FIELD_EPS0, c) for c in range(6)])
    e.close()
    lam, mu, n = p.lambda_, p.mu, 16
    assert np.abs(u.mean(axis=1)).max() <= 1e-12 * np.abs(u).max()
    tr = sig[0] + sig[1] + sig[2]
    eps = np.empty_like(sig)
    eps[:3] = (sig[:3] - lam / (3 * lam + 2 * mu) * tr) / (2 * mu)
    eps[3:] = sig[3:] / (2 * mu)  # tensor shear components
    eps += eps0
    f = np.fft.fftfreq(n)
    f0, f1, f2 = np.meshgrid(f, f, f, indexing="ij")
    k = [2 * np.pi * f2, 2 * np.pi * f1, 2 * np.pi * f0]  # x = axis 2, y = axis 1, z = axis 0
    mask = (np.abs(f0) < 0.5) & (np.abs(f1) < 0.5) & (np.abs(f2) < 0.5)
    mask[0, 0, 0] = False  # the mean strain is not a gradient
    U = [np.fft.fftn(u[a].reshape(n, n, n)) for a in range(3)]
    pairs = [(0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1)]  # xx yy zz yz xz xy
    scale = np.abs(eps - eps.mean(axis=1, keepdims=True)).max()
    for c, (a, b) in enumerate(pairs):
        grad = np.real(np.fft.ifftn(0.5j * (k[a] * U[b] + k[b] * U[a]) * mask))
        want = np.real(np.fft.ifftn(np.fft.fftn(eps[c].reshape(n, n, n)) * mask))
        assert np.abs(grad - want).max() <= 1e-9 * scale, c


# -------------------------------------------- spatially varying moduli
def test_inhomogeneous_solve_matches_reference(engine_lib):
    """The polarisation fixed point of a medium whose Lame moduli vary between
    0.7 and 1.3 of the uniform ones, against the reference's own
    InhomogeneousStressSolver on the same eigenstrain, moduli and mean strain
    (tests/golden/inhom_32.npz, generated from the reference's sources): the
    stress field and its mean to 1e-9 of the field's size."""
    g = golden("inhom_32")
    p = configs.ref2d(int(g["nx"]), int(g["ny"]), end="0.5", seed="5", soft="0")
    assert np.allclose([p.lambda_, p.mu], g["lame"], rtol=1e-15)
    e = api.Engine(p)
    for c in range(3):
        e.set_field(api.FIELD_EPS0, c, g["eps0"][c])
    e.set_field(api.FIELD_LAMBDA, 0, g["lam"])
    e.set_field(api.FIELD_MU, 0, g["mu"])
    e.set_mean_strain(list(g["epsavg"]))
    e.solve()
    sig = np.stack([e.field(api.FIELD_SIGMA, c) for c in range(3)])
    stress = np.array(e.scalars()["stress"][:3])
    e.close()
    scale = np.abs(g["sigma"]).max()
    assert np.abs(sig - g["sigma"]).max() <= 1e-9 * scale
    assert np.abs(stress - g["stress"]).max() <= 1e-9 * scale


def test_inhomogeneous_medium_steps(engine_lib):
    """The plain form steps with spatially varying moduli (every solve the
    fixed point); uniform moduli set explicitly leave the event sequence of the
    uniform medium unchanged."""
    def run(moduli):
        p = configs.ref2d(32, 32, end="0.5", seed="5", soft="0")
        e = api.Engine(p)
        if moduli is not None:
            lam, mu = moduli(p)
            e.set_field(api.FIELD_LAMBDA, 0, lam)
            e.set_field(api.FIELD_MU, 0, mu)
        e.run(max_events=30)
        ev, sc = e.events(), e.scalars()
        e.close()
        return ev, sc
    n = 32 * 32
    ev0, sc0 = run(None)
    ev1, sc1 = run(lambda p: (np.full(n, p.lambda_), np.full(n, p.mu)))
    for k in ("step", "kind", "site", "mode"):
        assert np.array_equal(ev0[k], ev1[k]), k
    rng = np.random.default_rng(3)
    ev2, sc2 = run(lambda p: (p.lambda_ * rng.uniform(0.8, 1.2, n), p.mu * rng.uniform(0.8, 1.2, n)))
    assert sc2["status"] == 0 and sc2["kstep"] == 30
    assert np.all(np.isfinite(sc2["stress"]))
    assert not np.array_equal(ev0["site"], ev2["site"])


# ------------------------------------------------- fixed-point 3D rates
@pytest.mark.parametrize("shape,barrier", [
    ((2, 2, 2), None), ((6, 9, 12), None), ((16, 16, 16), None),   # one chunk and less, a ragged last chunk
    ((64, 72, 108), None), ((96, 96, 96), None),                  # two and four sites per thread
    ((6, 9, 12), 40.0), ((6, 9, 12), 1e4), ((6, 9, 12), -0.5),    # barriers outside the fixed point's range, below zero
])
def test_fixed_point_rates_match_fp64_rates(engine_lib, shape, barrier):
    """The total rate of a step against the sum over all sites and modes of
    vt exp(-Q/kT) in extended precision, Q read back from the engine (its FP64
    chain, which the fixed-point pass does not use), under a stress field of
    about 1 GPa. Q carries a few roundings of 2^-53 of a few eV, 3e-14 of a
    rate at 455 K (kT = 0.039 eV); the bar is 1e-13. A barrier out of range
    sends its chunk through the FP64 chain; a negative one is an avalanche."""
    p = configs.stress32(n=shape[2])
    p.n[0], p.n[1], p.n[2] = shape
    eng = api.Engine(p)
    rng = np.random.default_rng(7)
    for c in range(6):
        eng.set_field(api.FIELD_EPS0, c, rng.standard_normal(eng.N) * 0.006)
    if barrier is not None:
        dF = eng.field(api.FIELD_DF)
        dF[eng.N // 2] = barrier
        eng.set_field(api.FIELD_DF, 0, dF)
    eng.solve()
    kT = p.temperature * 1.380658e-23 / 1.60217733e-19
    R = np.longdouble(0)
    neg = 0
    for m in range(20):
        Q = eng.field(api.FIELD_Q, m)
        neg += int((Q < 0).sum())
        R += np.exp(-Q.astype(np.longdouble) / np.longdouble(kT)).sum()
    R *= np.longdouble(p.voxel_volume * p.trial_frequency)
    eng.run(max_steps=1)
    ev, sc = eng.events(), eng.scalars()
    assert (sc["astep"] == 1) == (neg > 0)
    if neg == 0:
        assert abs(ev["total_rate"][0] / R - 1) < 1e-13
    eng.close()


# ------------------------------------------------- fixed-point solve
def _noalloc(lib, dim, shape, lam, mu, eps, ebar):
    import ctypes as C
    torch = pytest.importorskip("torch")
    d = torch.tensor(eps, dtype=torch.float64, device="cuda")
    s = torch.full_like(d, 7.0)
    eb = (C.c_double * len(ebar))(*ebar)
    st = lib.stz_solve_noalloc(dim, *shape, lam, mu, d.data_ptr(), eb, s.data_ptr(), None)
    assert st == api.OK, lib.stz_last_error().decode()
    return s.cpu().numpy()


@pytest.mark.parametrize("shape", [
    (2, 2, 2), (2, 3, 4), (1, 2, 2), (1, 1, 2), (3, 1, 6), (1, 512, 2), (2, 2, 512), (64, 2, 54),
    (1, 1024, 32), (1, 32, 1024), (2, 16, 648), (27, 9, 18),   # long lines: the passes' general forms
])
def test_fixed_point_solve_edges(engine_lib, oracle_lib, shape):
    """The solve in fixed point on lines of one value up to 1024, odd lengths and
    tiles with idle lanes, against the oracle's complex FP64 solve (the bar of
    test_fft_green_solve_matches_oracle)."""
    dim = 2 if shape[0] == 1 else 3
    p = configs.ref2d(shape[1], shape[2]) if dim == 2 else configs.shear64(seed=2)
    p.n[0], p.n[1], p.n[2] = shape
    ora = oracle_lib.Model(p)
    nc, N = 3 * (dim - 1), int(np.prod(shape))
    rng = np.random.default_rng(11)
    eps = rng.standard_normal((nc, N)) * 0.02
    for c in range(nc):
        ora.set_field(api.FIELD_EPS0, c, eps[c])
    ora.solve()
    want = np.stack([ora.field(api.FIELD_SIGMA, c) for c in range(nc)])
    ebar = ora.scalars()["eps_avg"][:nc]
    got = _noalloc(engine_lib, dim, shape, p.lambda_, p.mu, eps, ebar)
    assert rel_err(got, want) < 1e-11


@pytest.mark.parametrize("scale", [1e-200, 1e-30, 1e30, 1e200])
def test_fixed_point_solve_is_scale_free(engine_lib, scale):
    """A power of ten times the eigenstrain gives that times the stress to a few
    roundings, inside and outside the range of the FP32 line sums."""
    shape = (6, 8, 12)
    rng = np.random.default_rng(3)
    eps = rng.standard_normal((6, 576)) * 0.02
    a = _noalloc(engine_lib, 3, shape, 80.0, 35.0, eps, [0.0] * 6)
    b = _noalloc(engine_lib, 3, shape, 80.0, 35.0, eps * scale, [0.0] * 6) / scale
    assert np.abs(a - b).max() <= 1e-14 * np.abs(a).max()
    assert not _noalloc(engine_lib, 3, shape, 80.0, 35.0, eps * 0.0, [0.0] * 6).any()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_fixed_point_solve_keeps_nan(engine_lib, bad):
    """A value that is not finite makes every site's stress NaN, as it does in
    FP64 arithmetic (it enters every wave vector)."""
    eps = np.zeros((6, 16 * 12 * 8))
    eps[2, 77] = bad
    assert np.isnan(_noalloc(engine_lib, 3, (16, 12, 8), 80.0, 35.0, eps, [0.0] * 6)[2]).all()


@pytest.mark.parametrize("lam", [-30.0, 0.0, 35.0, 8000.0, 1e6])
def test_solve_for_extreme_media(engine_lib, oracle_lib, lam):
    """Lame constants at the ends of the fixed point's range and (1e6) beyond
    it, where the FP64 passes run. The rounding of FP64 grows with lambda / mu."""
    p = configs.shear64(seed=2, n=8)
    p.lambda_, p.mu = lam, 35.0
    ora = oracle_lib.Model(p)
    rng = np.random.default_rng(5)
    eps = rng.standard_normal((6, 512)) * 0.02
    for c in range(6):
        ora.set_field(api.FIELD_EPS0, c, eps[c])
    ora.solve()
    want = np.stack([ora.field(api.FIELD_SIGMA, c) for c in range(6)])
    got = _noalloc(engine_lib, 3, (8, 8, 8), lam, 35.0, eps, ora.scalars()["eps_avg"])
    assert rel_err(got, want) < 1e-11 * max(1.0, abs(lam) / 35.0)


# ------------------------------------------------- fixed-point 2D rates
@pytest.mark.parametrize("shape,scheme,mro,odd", [
    ((16, 18), api.SF_SQUARE_FWD, 0.0, None), ((48, 54), api.SF_LINEAR_FWD, 0.15, None),
    ((48, 54), api.SF_LINEAR_BWD, 0.0, None), ((48, 54), api.SF_EVEN, 0.0, None),
    ((48, 54), api.SF_CUBIC_FWD, 0.15, None), ((48, 54), api.SF_GAUSS_FWD, 0.0, None),
    ((576, 576), api.SF_SQUARE_FWD, 0.15, None), ((768, 1024), api.SF_SQUARE_FWD, 0.0, None),  # two, four sites a thread
    ((48, 54), api.SF_SQUARE_FWD, 0.0, "trace"), ((48, 54), api.SF_SQUARE_FWD, 0.0, "mode"),
    ((48, 54), api.SF_SQUARE_FWD, 0.0, "barrier"), ((48, 54), api.SF_SQUARE_FWD, 0.0, "soft"),
    ((48, 54), api.SF_SQUARE_FWD, 0.0, "hardened"),
])
def test_fixed_point_2d_rates_match_fp64_rates(engine_lib, shape, scheme, mro, odd):
    """The total rate of a step of the 2D model, half of its sites softened,
    against the sum of vt exp(-Q/kT) in extended precision over the engine's own
    FP64 Q's. Q carries a few roundings of 2^-52 of 2 eV and kT is 0.026 eV, so
    rates differ by some 1e-13; the bar is 3e-13. `odd`: one value outside the
    fixed point's range (a mode with a trace, one of strain above 1, a barrier
    of 30 eV, softening above 8, negative softening), whose chunk takes the FP64
    chain."""
    p = configs.ref2d(*shape, xfrac=mro, xq0="1.8")
    p.sf_scheme = scheme
    eng = api.Engine(p)
    N, rng = eng.N, np.random.default_rng(5)
    for c in range(3):
        eng.set_field(api.FIELD_EPS0, c, rng.standard_normal(N) * 0.004)
    hit = rng.random(N) < 0.5
    pd = np.where(hit, 0.07 * rng.standard_normal((2, N)), 0.0)
    soft = np.where(hit, np.minimum(p.perm_soft_cap, 26 * (pd ** 2).sum(0)), 0.0)
    if odd in ("soft", "hardened"):
        soft[N // 3] = 9.0 if odd == "soft" else -0.01
    for c, v in ((0, pd[0]), (1, -pd[0]), (2, pd[1])):
        eng.set_field(api.FIELD_PREV_DEPS, c, v)
    eng.set_field(api.FIELD_PERM_SOFT, 0, soft)
    eng.set_field(api.FIELD_TEMP_SOFT, 0, np.where(hit, 0.3, 0.0) * (rng.random(N) < 0.3))
    eng.set_field(api.FIELD_TLAST, 0, -p.t_temp * rng.uniform(0, 900, N))
    if odd in ("trace", "mode"):
        d = eng.field(api.FIELD_DEPS, 3 * 7)
        d[N // 2] = 0.01 if odd == "trace" else 1.5
        eng.set_field(api.FIELD_DEPS, 3 * 7, d)
        if odd == "mode":
            eng.set_field(api.FIELD_DEPS, 3 * 7 + 1, -d)
    if odd == "barrier":
        q = eng.field(api.FIELD_DF, 4)
        q[N // 2] = 30.0
        eng.set_field(api.FIELD_DF, 4, q)
    eng.solve()
    kT = p.temperature * 1.380658e-23 / 1.60217733e-19
    R, neg = np.longdouble(0), 0
    for m in range(20):
        Q = eng.field(api.FIELD_Q, m)
        neg += int((Q < 0).sum())
        R += np.exp(-Q.astype(np.longdouble) / np.longdouble(kT)).sum()
    R *= np.longdouble(p.voxel_volume * p.trial_frequency)
    eng.run(max_steps=1)
    ev, sc = eng.events(), eng.scalars()
    assert (sc["astep"] == 1) == (neg > 0)
    if neg == 0:
        assert abs(ev["total_rate"][0] / R - 1) < 3e-13
    eng.close()


@pytest.mark.parametrize("form", ["ref2d", "incremental", "mixed"])
@pytest.mark.parametrize("cap", [0, 256])
def test_runs_of_any_length_join(engine_lib, form, cap):
    """A run in parts that take every size of launch (one step, the graphs, a
    whole turn and its remainders) and one run of the same length give the same
    events and the same state, with the default ring of log entries and with a
    ring that wraps."""
    p = configs.ref2d(36, 48) if form == "ref2d" else configs.shear64(n=24)
    if form != "ref2d":
        p.solver = api.SOLVER_KERNEL
    if form == "mixed":
        p.precision = api.PREC_MIXED
    p.log_capacity = cap
    one, parts = api.Engine(p), api.Engine(p)
    lengths = [1, 1, 3, 5, 16, 17, 33, 64, 65, 129, 1]
    one.run(max_steps=sum(lengths))
    for n in lengths:
        parts.run(max_steps=n)
        assert len(parts.events()) == parts.scalars()["n_events_logged"]
    a, b = one.scalars(), parts.scalars()
    assert a["step"] == b["step"] == sum(lengths)
    assert a["n_events_logged"] == b["n_events_logged"]
    assert a["log_dropped"] == b["log_dropped"] == 0
    assert (one.events() == parts.events()).all()
    for k in ("time", "kstep", "astep"):
        assert a[k] == b[k]
    assert (one.field(api.FIELD_SIGMA, 0) == parts.field(api.FIELD_SIGMA, 0)).all()
    one.close()
    parts.close()


@pytest.mark.parametrize("shape", [(3, 4, 6), (2, 2, 2), (9, 3, 4), (4, 27, 8), (16, 6, 18), (12, 32, 24)])
@pytest.mark.parametrize("shift", [0.0, 1e-9, 2e-3])
def test_octant_update_is_the_solve(engine_lib, shape, shift):
    """The 3D incremental field after 12 events against the solve of the same
    eigenstrain and mean strain, on grids with even, odd and smallest axes.
    `shift`: the mean strain is moved by this much between the events, so that
    the updates carry a uniform stress from far below to far above the event's.
    An update rounds the field once (2^-53 of it) and its own sums at 2^-58;
    the solve's own error is some 1e-15 of the field: 12 updates stay below 1e-14."""
    p = api.default_params(api.MODEL_GLOBAL3D)
    p.n[0], p.n[1], p.n[2] = shape
    p.loading, p.solver, p.seed = api.LOAD_SHEAR, api.SOLVER_KERNEL, 3
    p.strain_rate, p.end_strain, p.strain_increment = 5e-5, 1.0, 1e9
    eng = api.Engine(p)
    for i in range(12):
        if shift:
            sc = eng.scalars()
            eng.set_mean_strain([e + shift * (-1) ** i * (c + 1) for c, e in enumerate(sc["eps_avg"])])
        eng.run(max_events=1)
    # the strain that loading added after the last event is not in the field yet
    a = [eng.field(api.FIELD_SIGMA, c) for c in range(6)]
    eng.solve()
    b = [eng.field(api.FIELD_SIGMA, c) for c in range(6)]
    size = max(np.abs(v).max() for v in b)
    for c in range(6):
        d = a[c] - b[c]
        assert np.abs(d - d.mean()).max() < 1e-14 * size
    eng.close()


@pytest.mark.parametrize("odd", [None, "mode"])
@pytest.mark.parametrize("shape", [(72, 96), (162, 192), (192, 216)])
def test_split_2d_rates_match_fp64_rates(engine_lib, shape, odd):
    """The same on grids whose blocks' modes are split into four, two and one
    parts (up to 76, 152 and more blocks of 256 sites on 152 multiprocessors);
    `odd`: a value that sends one part of a block through the FP64 chain."""
    test_fixed_point_2d_rates_match_fp64_rates(engine_lib, shape, api.SF_SQUARE_FWD, 0.0, odd)


@pytest.mark.parametrize("shape", [(36, 36, 36), (48, 48, 54)])
def test_split_3d_rates_match_fp64_rates(engine_lib, shape):
    """The 3D rates in two parts and in one (up to 228 and more blocks)."""
    test_fixed_point_rates_match_fp64_rates(engine_lib, shape, None)


FLAT = [(1, 8, 12), (1, 1, 2), (1, 16, 16), (1, 9, 6), (1, 64, 48)]


@pytest.mark.parametrize("shape", FLAT)
def test_flat_3d_grid_solves(engine_lib, oracle_lib, shape):
    """Six components on a grid without an axis 0: the context's solve and the
    stand-alone one against the oracle's (the bar of
    test_fft_green_solve_matches_oracle)."""
    p = configs.shear64(seed=2)
    p.n[0], p.n[1], p.n[2] = shape
    eng, ora = api.Engine(p), oracle_lib.Model(p)
    rng = np.random.default_rng(11)
    eps = rng.standard_normal((6, eng.N)) * 0.02
    for c in range(6):
        eng.set_field(api.FIELD_EPS0, c, eps[c])
        ora.set_field(api.FIELD_EPS0, c, eps[c])
    eng.solve()
    ora.solve()
    want = np.stack([ora.field(api.FIELD_SIGMA, c) for c in range(6)])
    assert rel_err(np.stack([eng.field(api.FIELD_SIGMA, c) for c in range(6)]), want) < 1e-11
    got = _noalloc(engine_lib, 3, shape, p.lambda_, p.mu, eps, ora.scalars()["eps_avg"])
    assert rel_err(got, want) < 1e-11
    eng.close()


@pytest.mark.parametrize("shape", FLAT[:1] + FLAT[2:3])
@pytest.mark.parametrize("form", ["incremental", "mixed"])
def test_flat_3d_grid_updates(engine_lib, oracle_lib, shape, form):
    """The updates and the FP64 re-solve on such a grid: the field after 12
    events against the oracle's solve of the same eigenstrain and mean strain;
    bars of the octant test (FP64) and of the mixed form (1e-5)."""
    p = configs.shear64(seed=2, eng_end=1e9)
    p.n[0], p.n[1], p.n[2] = shape
    p.solver = api.SOLVER_KERNEL
    if form == "mixed":
        p.precision, p.resolve_period, p.resolve_fp64 = api.PREC_MIXED, 5, 1
    eng, ora = api.Engine(p), oracle_lib.Model(p)
    eng.run(max_events=12)
    sc = eng.scalars()
    for c in range(6):
        ora.set_field(api.FIELD_EPS0, c, eng.field(api.FIELD_EPS0, c))
    if form == "mixed":
        assert sc["n_resolves"] == 2 and sc["stress_err_max_worst"] < 1e-5
    ora.solve()
    which, comps, bar = (api.FIELD_SDEV, 5, 1e-5) if form == "mixed" else (api.FIELD_SIGMA, 6, 1e-13)
    want = np.stack([ora.field(api.FIELD_SIGMA, c) for c in range(6)])
    if form == "mixed":
        r2, r6 = 0.5 ** 0.5, 6 ** -0.5
        want = np.stack([(want[0] - want[1]) * r2, (2 * want[2] - want[0] - want[1]) * r6, *(want[3:] / r2)])
    for c in range(comps):
        d = eng.field(which, c) - want[c]  # up to the uniform stress of the loading
        assert np.abs(d - d.mean()).max() < bar * np.abs(want).max()
    eng.close()


@pytest.mark.parametrize("precision", [api.PREC_FP64, api.PREC_MIXED])
@pytest.mark.parametrize("shape", [(256, 16, 32), (256, 32, 64), (512, 16, 16), (1024, 2, 8)])
def test_correlated_barriers_on_long_axis_0(engine_lib, shape, precision):
    """The barrier filter where axis 0 is longer than axis 1, whatever tile the
    tuner took for axis 1: neighbours a site apart along axis 0 have the
    Gaussian covariance's correlation, exp(-1/32) = 0.969 for a length of 4
    sites (0.01 over a few hundred independent patches; without a filter along
    the axis it is 0 to 0.06), and the context runs."""
    p = configs.shear64(seed=3, eng_end=1e9)
    p.n[0], p.n[1], p.n[2] = shape
    p.df_kind, p.q0_sd, p.q0_corr_len, p.precision = api.DF_CORRELATED, 0.15, 4.0, precision
    p.solver = api.SOLVER_KERNEL if precision == api.PREC_MIXED else api.SOLVER_FFT
    eng = api.Engine(p)
    q = eng.field(api.FIELD_DF).reshape(shape)
    q = q - q.mean()
    assert (q * np.roll(q, 1, 0)).mean() / (q * q).mean() > 0.93
    eng.run(max_events=2)
    assert eng.scalars()["kstep"] == 2
    eng.close()


@pytest.mark.parametrize("shape", [(1, 2, 5832), (1, 16, 8192), (2, 2, 3888), (2, 2, 4096), (2, 4, 8192)])
def test_contexts_of_long_lines(engine_lib, oracle_lib, shape):
    """Lines up to the longest accepted, 8192 values, where the passes hold one
    line a block: the solve against the oracle's (the bar of
    test_fft_green_solve_matches_oracle), and steps. In 2D without the wave
    number that is Nyquist's on both axes: the reference's s - round(s) takes
    either sign there, as (n/2)(1/n) rounds to 1/2 or, for 5832, to less."""
    p = configs.ref2d(shape[1], shape[2]) if shape[0] == 1 else configs.shear64(seed=2)
    p.n[0], p.n[1], p.n[2] = shape
    eng, ora = api.Engine(p), oracle_lib.Model(p)
    rng = np.random.default_rng(11)
    for c in range(eng.nc):
        v = rng.standard_normal(eng.N) * 0.02
        eng.set_field(api.FIELD_EPS0, c, v)
        ora.set_field(api.FIELD_EPS0, c, v)
    eng.solve()
    ora.solve()
    alt = 1.0 - 2.0 * (np.indices(shape).sum(0).ravel() % 2)
    for c in range(eng.nc):
        want = ora.field(api.FIELD_SIGMA, c)
        d = eng.field(api.FIELD_SIGMA, c) - want
        if shape[0] == 1:
            d -= alt * (alt * d).mean()
        assert np.abs(d).max() < 1e-11 * np.abs(want).max()
    eng.run(max_steps=2)
    assert eng.scalars()["step"] == 2
    eng.close()


@pytest.mark.parametrize("shape", [(1, 2, 4096), (1, 32, 6144), (2, 2, 4096), (2, 2, 6144)])
@pytest.mark.parametrize("lam", [80.0, 1e6])
def test_noalloc_solves_of_long_lines(engine_lib, oracle_lib, shape, lam):
    """Lines whose tables fill the fixed scratch, in fixed point and (lambda of
    1e6) in FP64, against the oracle (the bars of test_solve_for_extreme_media)."""
    dim = 2 if shape[0] == 1 else 3
    p = configs.ref2d(shape[1], shape[2]) if dim == 2 else configs.shear64(seed=2)
    p.n[0], p.n[1], p.n[2] = shape
    p.lambda_, p.mu = lam, 35.0
    ora = oracle_lib.Model(p)
    nc = 3 * (dim - 1)
    eps = np.random.default_rng(11).standard_normal((nc, int(np.prod(shape)))) * 0.02
    for c in range(nc):
        ora.set_field(api.FIELD_EPS0, c, eps[c])
    ora.solve()
    want = np.stack([ora.field(api.FIELD_SIGMA, c) for c in range(nc)])
    got = _noalloc(engine_lib, dim, shape, lam, 35.0, eps, ora.scalars()["eps_avg"][:nc])
    assert rel_err(got, want) < 1e-11 * max(1.0, lam / 35.0)


def _solve_extended(shape, lam, mu, eps):
    """The solve for a zero mean strain in extended precision (numpy's long
    double transforms); on Nyquist planes the average over the components' signs
    (3D: each for itself, 2D: together)."""
    ld, nc = np.longdouble, len(eps)
    d = 2 if nc == 3 else 3
    at = [(0, 0), (1, 1), (0, 1)] if nc == 3 else [(0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1)]
    lam, mu = ld(lam), ld(mu)

    def stress(e):
        s = 2 * mu * e
        s[:d] += lam * e[:d].sum(0)
        return s
    E = np.stack([np.fft.fftn(e.reshape(shape).astype(np.clongdouble)) for e in eps])
    k = [np.arange(n).reshape([-1 if i == a else 1 for i in range(3)]) for a, n in enumerate(shape)]
    w = [np.where(2 * i < n, i, i - n).astype(ld) / n if n > 1 else ld(0) * i for i, n in zip(k, shape)][::-1]
    ny = [(2 * i == n) & (n > 1) for i, n in zip(k, shape)][::-1]
    norm = np.sqrt(w[0] ** 2 + w[1] ** 2 + w[2] ** 2)
    norm[0, 0, 0] = 1
    t = {ab: v for v, ab in zip(stress(E.copy()), at)}
    t.update({(b, a): v for (a, b), v in t.items()})
    flips = (0, 7) if nc == 3 else range(8)
    out = 0
    for sg in flips:
        g = [np.where(ny[a] & bool(sg >> a & 1), -w[a], w[a]) / norm for a in range(3)]
        F = [sum(t[a, b] * g[b] for b in range(d)) for a in range(d)]
        G = sum(g[a] * F[a] for a in range(d))
        out = out + stress(np.stack([(F[a] * g[b] + F[b] * g[a]) / (2 * mu) - (lam + mu) / (lam + 2 * mu) / mu * G *
                                     g[a] * g[b] for a, b in at]) - E)
    return np.stack([np.fft.ifftn(c / len(flips)).real for c in out]).reshape(nc, -1)


@pytest.mark.parametrize("shape", [(1, 512, 64), (1, 1024, 16), (1, 128, 512), (512, 8, 16)])
def test_solve_of_nearly_uniform_eigenstrain(engine_lib, shape):
    """A uniform eigenstrain with 10% of spread, whose k = 0 term is a hundred
    times the other terms of its column: the stress within 2.5e-16 (relative L2)
    of the solve in extended precision. Its values are stored to 2^-53, which
    alone is 0.6e-16, and FP64 passes come to 1.4e-16 to 1.9e-16."""
    nc = 3 if shape[0] == 1 else 6
    eps = 0.05 * (1 + 0.1 * np.random.default_rng(5).standard_normal((nc, int(np.prod(shape)))))
    want = _solve_extended(shape, 80.0, 35.0, eps)
    d = _noalloc(engine_lib, 2 if nc == 3 else 3, shape, 80.0, 35.0, eps, [0.0] * nc) - want
    assert np.sqrt((d ** 2).sum() / (want ** 2).sum()) < 2.5e-16


@pytest.mark.parametrize("shape", [(8, 12, 16), (1, 16, 64), (1, 9, 8)])
def test_solve_at_the_scales_limits(engine_lib, shape):
    """Fields whose partial sums reach a line's sum of magnitudes, the bound its
    integer scale is taken from: uniform, alternating, one wave in equal sine and
    cosine parts along every axis, one site; at 32 amplitudes of an octave, so
    that the sums lie everywhere up to the scale's limit. 1e-13 of the largest
    stress: an overflow is of its own size."""
    nc = 3 if shape[0] == 1 else 6
    ph = [2 * np.pi * i / n for i, n in zip(np.indices(shape), shape)]
    alt = (-1.0) ** np.indices(shape).sum(0)
    delta = np.zeros(shape)
    delta[0, 1 % shape[1], 2] = 1.0
    fields = [np.ones(shape), alt, delta] + [np.cos(k * x + np.pi / 4) for x in ph for k in (1, 2)]
    for sign in (1.0, -1.0):
        for v in fields:
            eps = np.stack([v.ravel() * (sign if c % 2 else 1.0) for c in range(nc)])
            want = _solve_extended(shape, 80.0, 35.0, eps).astype(float)
            size = np.abs(want).max()
            for j in range(32):
                a = 2.0 ** (j / 32)
                got = _noalloc(engine_lib, 2 if nc == 3 else 3, shape, 80.0, 35.0, eps * a, [0.0] * nc)
                assert np.abs(got - a * want).max() < 1e-13 * a * max(size, 1.0)


def _dense_error(lib, shape):
    nc = 3 if shape[0] == 1 else 6
    eps = 0.05 * np.random.default_rng(5).standard_normal((nc, int(np.prod(shape))))
    want = _solve_extended(shape, 80.0, 35.0, eps)
    d = _noalloc(lib, 2 if nc == 3 else 3, shape, 80.0, 35.0, eps, [0.0] * nc) - want
    return np.sqrt((d ** 2).sum() / (want ** 2).sum())


@pytest.mark.parametrize("shape", [(2, 2, 1024), (4, 4, 1024), (1024, 2, 16)])
def test_dense_lines_of_a_thousand_values(engine_lib, shape):
    """Random eigenstrain on long lines, whose values lie lowest above the
    integers' unit: within 1e-15 (relative L2) of the solve in extended
    precision, where FP64 passes come to 0.8e-15 to 0.9e-15."""
    assert _dense_error(engine_lib, shape) < 1e-15


@pytest.mark.parametrize("shape", [(2, 2, 4096), (4, 2, 1728), (1, 16, 6144), (1, 16, 1296)])
def test_dense_lines_of_thousands_of_values(engine_lib, shape):
    """Lines on both sides of the longest that the fixed-point passes take: as
    near to extended precision as FP64 passes, 0.8e-15 to 0.9e-15 (six
    components) and 1.1e-15 (three)."""
    assert _dense_error(engine_lib, shape) < (1e-15 if shape[0] > 1 else 1.2e-15)


@pytest.mark.parametrize("n2", [1458, 2916])
def test_nyquist_sign_of_the_reference(engine_lib, oracle_lib, n2):
    """Lengths whose (n/2)(1/n) rounds below 1/2, so that the reference's
    s - round(s) gives the Nyquist number its positive sign: with Nyquist's on
    axis 1 the 2D operator depends on it. Against the oracle, which forms it so
    (the bar of test_fft_green_solve_matches_oracle)."""
    p = configs.ref2d(16, n2)
    eng, ora = api.Engine(p), oracle_lib.Model(p)
    rng = np.random.default_rng(11)
    for c in range(3):
        v = rng.standard_normal(eng.N) * 0.02
        eng.set_field(api.FIELD_EPS0, c, v)
        ora.set_field(api.FIELD_EPS0, c, v)
    eng.solve()
    ora.solve()
    for c in range(3):
        assert rel_err(eng.field(api.FIELD_SIGMA, c), ora.field(api.FIELD_SIGMA, c)) < 1e-11
    eng.close()


def test_fixed_point_rates_under_two_large_stresses(engine_lib):
    """A field stress and a uniform stress of the same sign, each within the
    fixed point's limit of 2^(8 - L) GPa and their sum beyond it, against a mode
    whose rate argument they take below the representable 2^-1022: the FP64
    chain's total rate and no avalanche. Barriers of 14 eV, Q to some 1e-15 of
    them, 1e-12 of a rate at kT = 0.039 eV."""
    p = configs.stress32(seed=58, n=4)
    p.applied_stress[api.XY] = 0.0
    kT = p.temperature * 1.380658e-23 / 1.60217733e-19
    eng = api.Engine(p)
    Q = np.empty((7, 20))
    for k in range(7):
        for c in range(6):
            eng.set_field(api.FIELD_SIGMA, c, np.full(eng.N, float(c == k - 1)))
        Q[k] = [eng.field(api.FIELD_Q, m)[0] for m in range(20)]
    eng.close()
    G = (Q[0] - Q[1:]).T * np.log2(np.e) / kT  # work of each mode per GPa, in powers of two
    # the modes' largest sum of coefficients just below a power of two, 2^L
    size = np.abs(G[:, [0, 1, 3, 4, 5]]).sum(1).max()
    L = int(np.ceil(np.log2(size)))
    p.voxel_volume *= 0.999 * 2.0 ** L / size
    stress = -np.sign(G[18]) * 0.97 * 2.0 ** (8 - L)
    for c in range(6):
        p.applied_stress[c] = stress[c]
    eng = api.Engine(p)
    eng.set_mean_strain([0.0] * 6)
    eng.solve()
    eng.run(max_events=1)  # the uniform stress now makes up for the applied one
    for c in range(6):
        eng.set_field(api.FIELD_SIGMA, c, np.full(eng.N, stress[c]))
    y0 = 524 - 1022 - np.log2(p.voxel_volume * p.trial_frequency)
    eng.set_field(api.FIELD_DF, 0, np.full(eng.N, -y0 * kT / np.log2(np.e)))
    Q = np.stack([eng.field(api.FIELD_Q, m) for m in range(20)])
    assert Q.min() > 0 and Q[18].min() * np.log2(np.e) / kT > 1070
    R = np.longdouble(p.voxel_volume * p.trial_frequency) * np.exp(-Q.astype(np.longdouble) / np.longdouble(kT)).sum()
    eng.run(max_steps=1)
    assert eng.scalars()["astep"] == 0
    assert abs(eng.events()["total_rate"][-1] / R - 1) < 1e-12
    eng.close()


@pytest.mark.parametrize("shape", [(3, 4, 6), (12, 32, 24)])
@pytest.mark.parametrize("shift", [1e-9, 2e-3])
def test_octant_update_carries_the_uniform_stress(engine_lib, shape, shift):
    """test_octant_update_is_the_solve with the field's mean: without the
    subtracted error and under shear the strain that loading adds after an event
    is 2 mu of it in the uniform stress, so the whole field, moved by C: of the
    mean strain's changes between the events, is the solve's (the same bar)."""
    p = api.default_params(api.MODEL_GLOBAL3D)
    p.n[0], p.n[1], p.n[2] = shape
    p.loading, p.solver, p.seed, p.no_subtract_error = api.LOAD_SHEAR, api.SOLVER_KERNEL, 3, 1
    p.strain_rate, p.end_strain, p.strain_increment = 5e-5, 1.0, 1e9
    eng = api.Engine(p)
    for i in range(12):
        sc = eng.scalars()
        eng.set_mean_strain([e + shift * (-1) ** i * (c + 1) for c, e in enumerate(sc["eps_avg"])])
        eng.run(max_events=1)
    a = [eng.field(api.FIELD_SIGMA, c) for c in range(6)]
    eng.solve()
    b = [eng.field(api.FIELD_SIGMA, c) for c in range(6)]
    size = max(np.abs(v).max() for v in b)
    assert size > 1e-2
    for c in range(6):
        assert np.abs(a[c] - b[c]).max() < 1e-14 * size
    eng.close()

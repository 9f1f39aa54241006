"""The workloads that performance work on this package is measured on.

Each case is one call, or the few calls of one step, of the public Python
interface (fjmodels_gb300) on the model families, grids and quadrature rules of
the tests, the benchmark and the README: the Legendre projection and radial
Poisson solve, the potential and action batches, the plain FP64 and the mixed
phase-space moments, line-of-sight profiles, a batch of models, the action
surrogate and a restarted self-consistent model.

listed() names the cases, draw(rng) gives more of the same ranges, prepare()
makes what a caller holds before the call, run() makes one pass and returns
everything it computes, work() says what a pass cannot do without, and exact()
gives the outputs in extended precision where they have a closed form.
"""
import math

import numpy as np
import torch

import fjmodels_gb300 as F
from fjmodels_gb300 import _abi as A

TPI = 6.283185307179586
# The reference's algorithm, operations tallied by the instrumented oracle on
# the rotating NFW 80x40 model: per phase-space evaluation of a 22-point rule
# (39 % of the nodes bound), and per bound orbit.
FLOPS_PER_NODE = 1.33e5
FLOPS_PER_ORBIT = FLOPS_PER_NODE / 0.39

# the radial range of each family in units of its scale radius (tests, benchmark)
RANGE = {"Hernquist": (0.01, 100.0), "Isochrone": (0.01, 100.0), "NFW": (1e-3, 300.0)}
KINDS = {"line": A.FJ_LOS_LINE, "vphi": A.FJ_LOS_PVPHI, "vz": A.FJ_LOS_PVZ, "vr": A.FJ_LOS_PVR}


def listed():
    return [
        # The multipole half of every iteration on the first configuration's
        # 40x20 grid: microseconds of work, so launches and latency count.
        {"name": "multipoles_40x20", "do": "multipoles", "model": "Hernquist", "nr": 40, "ngauss": 20, "npoly": 5,
         "poisson": "cumulative"},
        # The reference's adaptive radial integrals (the default Poisson solve)
        # on the 80-radius, l <= 12 model.
        {"name": "poisson_adaptive_80x7", "do": "multipoles", "model": "NFW", "nr": 80, "ngauss": 40, "npoly": 7,
         "poisson": "adaptive"},
        # Potential and forces along many test orbits or on a plotting grid.
        {"name": "potential_200k", "do": "potential", "model": "NFW", "nr": 80, "npoly": 7, "n": 200_003},
        # Actions of a catalogue of stars in a model's potential.
        {"name": "actions_20k", "do": "actions", "model": "Hernquist", "nr": 40, "npoly": 5, "n": 20_001},
        # Moments at a handful of observed positions, plain FP64 with the
        # default rule: too few blocks to fill the chip.
        {"name": "points_fp64_6", "do": "points", "model": "Isochrone", "nr": 40, "npoly": 5, "n": 6, "nq": 22,
         "rule": "reference", "precision": "fp64"},
        # One plain FP64 iteration (the default precision, parity with the
        # reference) of the small model the tests compare with the oracle.
        {"name": "iteration_fp64_16x6", "do": "iteration", "model": "Hernquist", "nr": 16, "ngauss": 6, "npoly": 3,
         "nq": 22, "rule": "reference", "precision": "fp64", "poisson": "adaptive"},
        # Line-of-sight velocity profile of a converged model, some velocities
        # of the reference's output file.
        {"name": "line_profile_40", "do": "los", "model": "NFW", "nr": 80, "npoly": 7, "kind": "line", "n": 40,
         "nq": 22, "rule": "tanhsinh"},
        # One mixed iteration of a small model, as a parameter search runs it.
        {"name": "iteration_mixed_24x8", "do": "iteration", "model": "Hernquist", "nr": 24, "ngauss": 8, "npoly": 4,
         "nq": 16, "rule": "tanhsinh", "precision": "mixed", "poisson": "adaptive"},
        # The headline configuration: one mixed iteration of the rotating NFW
        # model on the 80x40 grid, l <= 12, 22^3 velocity nodes.
        {"name": "iteration_mixed_80x40", "do": "iteration", "model": "NFW", "nr": 80, "ngauss": 40, "npoly": 7,
         "nq": 22, "rule": "tanhsinh", "precision": "mixed", "poisson": "cumulative"},
        # Many models of mixed sizes in one launch (a DF parameter study).
        {"name": "batch_mixed_6", "do": "batch", "models": 6, "nr": 40, "ngauss": 16, "npoly": 5, "nq": 16,
         "rule": "tanhsinh", "precision": "mixed"},
        # The action surrogate's tensor-core moments on the headline grid.
        {"name": "surrogate_80x40", "do": "surrogate", "model": "NFW", "nr": 80, "ngauss": 40, "npoly": 7, "nq": 22,
         "rule": "tanhsinh"},
        # A whole call: a model restarted from its tables and iterated on.
        {"name": "restart_mixed_33x11", "do": "restart", "model": "NFW", "nr": 33, "ngauss": 11, "npoly": 5, "nq": 14,
         "rule": "tanhsinh", "precision": "mixed", "iterations": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["multipoles", "potential", "actions", "points", "iteration", "iteration", "los", "batch",
                     "surrogate", "restart"])
    c = {"do": do, "model": rng.choice(sorted(RANGE)), "nr": _log_int(rng, 12, 96), "npoly": rng.randint(2, 9)}
    precision = rng.choice(["fp64", "mixed"])
    nq = 2 * rng.randint(5, 11)
    rule = "reference" if nq == 22 and rng.random() < 0.5 else "tanhsinh"
    if do == "multipoles":
        c.update(ngauss=rng.randint(4, 48), poisson=rng.choice(["cumulative", "adaptive"]))
    elif do == "potential":
        c.update(n=_log_int(rng, 1, 200_000))
    elif do == "actions":
        c.update(n=_log_int(rng, 1, 20_000))
    elif do == "points":
        n = _log_int(rng, 1, 40) if precision == "fp64" else _log_int(rng, 1, 2000)
        c.update(n=n, nq=nq, rule=rule, precision=precision)
    elif do == "iteration":
        most = 800_000 if precision == "fp64" else 20_000_000  # phase-space nodes of a pass
        c["nr"] = min(c["nr"], max(12, most // (4 * nq ** 3)))
        c.update(ngauss=max(2, min(rng.randint(4, 40), most // (c["nr"] * nq ** 3))), nq=nq, rule=rule,
                 precision=precision, poisson=rng.choice(["cumulative", "adaptive"]))
    elif do == "los":
        kind = rng.choice(sorted(KINDS))
        c.update(kind=kind, n=_log_int(rng, 1, 30 if kind == "line" else 300), nq=nq, rule=rule)
    elif do == "batch":
        c.pop("model")
        c.update(models=rng.randint(2, 9), nr=_log_int(rng, 12, 48), ngauss=rng.randint(4, 16),
                 npoly=rng.randint(2, 6), nq=2 * rng.randint(5, 8), rule="tanhsinh", precision="mixed")
    elif do == "surrogate":
        c.update(ngauss=rng.randint(4, 40), nq=nq, rule=rule, npoly=rng.randint(2, 8))
    else:
        c.update(nr=_log_int(rng, 12, 40), ngauss=rng.randint(4, 16), nq=2 * rng.randint(5, 8), rule="tanhsinh",
                 precision="mixed", iterations=rng.randint(2, 5))
    return c


# ------------------------------------------------------------------ inputs
def _seg(a, b, m, c0, c1):
    """int_a^b x^m (c0 + c1 x) dx"""
    t0 = np.log(b / a) if m == -1 else (b ** (m + 1) - a ** (m + 1)) / (m + 1)
    t1 = np.log(b / a) if m == -2 else (b ** (m + 2) - a ** (m + 2)) / (m + 2)
    return c0 * t0 + c1 * t1


def _solve(ar, rhl, dtype=np.longdouble):
    """Potential multipoles and their radial derivatives of the piecewise
    linear density multipoles rhl [nr][npoly], constant inside ar[0] and
    falling as r^-4 outside."""
    ar, rhl = np.asarray(ar, dtype), np.asarray(rhl, dtype)
    phil, Pr, Pr2 = (np.zeros_like(rhl) for _ in range(3))
    a, b = ar[:-1], ar[1:]
    for k in range(rhl.shape[1]):
        l = 2 * k
        y = rhl[:, k]
        s = (y[1:] - y[:-1]) / (b - a)
        c0 = y[:-1] - s * a
        inner = np.concatenate([[y[0] * ar[0] ** (l + 3) / (l + 3)], _seg(a, b, l + 2, c0, s)])
        outer = np.concatenate([_seg(a, b, 1 - l, c0, s), [max(y[-1], dtype(0)) * ar[-1] ** (2 - l) / (l + 2)]])
        Ii, Ie = np.cumsum(inner), np.cumsum(outer[::-1])[::-1]
        phil[:, k] = -TPI * (Ii / ar ** (l + 1) + Ie * ar ** l)
        Pr[:, k] = -TPI * (-(l + 1) * Ii / ar ** (l + 2) + l * Ie * ar ** (l - 1))
        Pr2[:, k] = -TPI * ((l + 2) * (l + 1) * Ii / ar ** (l + 3) + (l - 1) * l * Ie * ar ** (l - 2)
                            - (2 * l + 1) * y)
    return phil, Pr, Pr2


def _dev(x):
    return torch.tensor(np.ascontiguousarray(x, dtype=np.float64), device="cuda")


def _params(model, rng):
    """A seeded DF of the family: rotation, anisotropy, mass and scale."""
    g = lambda: float(rng.uniform(0.3, 1.2))  # noqa: E731
    return F.DFParams(model, dphi_h=g(), dz_h=g(), dphi_g=g(), dz_g=g(), chi=float(rng.uniform(0.0, 2.0)),
                      mass=float(10 ** rng.uniform(-0.3, 0.3)), r0=float(10 ** rng.uniform(-0.2, 0.2)), k=0.5)


def _tables(model, nr, npoly, rng):
    """A flattened model's DF, radii, density multipoles and potential tables."""
    df = _params(model, rng)
    lo, hi = RANGE[model]
    ar = F.log_grid(lo * df.r0, hi * df.r0, nr)
    rhl = F.guess_rhl(ar, 24, npoly, model, df.mass, df.r0, float(rng.uniform(0.6, 1.0)))
    return df, ar, rhl, [np.asarray(t, np.float64) for t in _solve(ar, rhl)]


def _model(ctx, model, nr, npoly, rng):
    df, ar, rhl, tabs = _tables(model, nr, npoly, rng)
    E, D, _ = F.tabulate_delta(ar, *tabs)
    return {"df": df, "ar": ar, "rhl": rhl, "tabs": tabs, "table": (E, D),
            "pot": ctx.potential(_dev(ar), *map(_dev, tabs)), "delta": ctx.delta(_dev(E), _dev(D))}


def _rule(case):
    prec = A.FJ_PREC_MIXED if case.get("precision") == "mixed" else A.FJ_PREC_FP64
    if case["rule"] == "reference":
        return F.Rule(precision=prec)
    return F.Rule(*F.tanh_sinh_rule(case["nq"]), precision=prec)


def _zeros(*shape):
    return torch.zeros(shape, dtype=torch.float64, device="cuda")


def _grids(case, ar, rng):
    """Moment grids [6][nr][ngauss] as an iteration leaves them: a density
    falling outwards, dispersions of order one, flattened and not smooth."""
    x = np.asarray(ar)[:, None] / ar[len(ar) // 2]
    g = np.exp(0.05 * rng.standard_normal((6, len(ar), case["ngauss"]))) / np.sqrt(1.0 + x)
    g[0] /= x * (1.0 + x) ** 2.5
    return g


def _points(ar, n, rng, wide):
    lo, hi = math.log(ar[0]), math.log(ar[-1])
    w = math.log(3.0) if wide else 0.0
    r = np.exp(rng.uniform(lo - w, hi + w, n))
    c = rng.uniform(0.01, 0.99, n) * (rng.choice([-1.0, 1.0], n) if wide else 1.0)
    return np.stack([r * np.sqrt(1.0 - c * c), r * c], 1)


def _escape(m, Rz):
    """Escape speed at points of a model, from the monopole alone (a scale for velocities)."""
    r = np.clip(np.hypot(Rz[:, 0], Rz[:, 1]), m["ar"][0], m["ar"][-1])
    return np.sqrt(-2.0 * np.interp(r, m["ar"], m["tabs"][0][:, 0]))


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 4099])
    ctx = F.Context(0)
    s = {"case": case, "ctx": ctx}
    do = case["do"]
    if case.get("poisson") == "cumulative" or do == "restart":
        ctx.set_poisson(A.FJ_POISSON_CUMULATIVE)
    if do == "batch":
        s["rule"], s["items"] = _rule(case), []
        for i in range(case["models"]):
            nr, ng = max(12, case["nr"] - 3 * i), max(3, case["ngauss"] - i)
            m = _model(ctx, sorted(RANGE)[i % 3], nr, case["npoly"], rng)
            s["items"].append((m["pot"], m["delta"], m["df"], ng, _zeros(6, nr, ng)))
        return s
    if do == "multipoles":
        df, ar, rhl, _ = _tables(case["model"], case["nr"], case["npoly"], rng)
        nr, npl = case["nr"], case["npoly"]
        s.update(ar=_dev(ar), grids=_dev(_grids(case, ar, rng)), coef=_zeros(6, nr, npl),
                 out=[_zeros(nr, npl) for _ in range(3)])
        return s
    m = _model(ctx, case["model"], case["nr"], case["npoly"], rng)
    s.update(m)
    nr, npl = case["nr"], case["npoly"]
    if do == "potential":
        s.update(Rz=_dev(_points(m["ar"], case["n"], rng, True)), out=_zeros(case["n"], 3))
    elif do == "actions":
        Rz = _points(m["ar"], case["n"], rng, True)
        v = rng.standard_normal((case["n"], 3)) * (0.35 * _escape(m, Rz))[:, None]
        s.update(pts=_dev(np.concatenate([Rz, v], 1)), out=_zeros(case["n"], 2))
    elif do == "points":
        s.update(rule=_rule(case), Rz=_dev(_points(m["ar"], case["n"], rng, False)), out=_zeros(6, case["n"]))
    elif do == "iteration":
        s.update(rule=_rule(case), grids=_zeros(6, nr, case["ngauss"]), coef=_zeros(6, nr, npl),
                 out=[_zeros(nr, npl) for _ in range(3)])
    elif do == "los":
        Rz = _points(m["ar"][nr // 4: -nr // 8], case["n"], rng, False)
        v = rng.uniform(-0.8, 0.8, case["n"])
        if case["kind"] != "line":  # a line profile's velocity is in units of the escape speed
            v = v * _escape(m, Rz)
        s.update(rule=_rule(case), Rzv=_dev(np.concatenate([Rz, v[:, None]], 1)), rhl_d=_dev(m["rhl"]),
                 out=_zeros(case["n"]))
    elif do == "surrogate":
        s.update(rule=_rule(case), net=F.Surrogate(ctx, batch=4096, seed=int(seed) % 1000003 + 1),
                 grids=_zeros(6, nr, case["ngauss"]))
    elif do == "restart":
        s.update(rule=_rule(case), tables=dict(zip(("ar", "phil", "Pr", "Pr2"), (m["ar"], *m["tabs"]))))
    else:
        raise ValueError(do)
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    do = case["do"]
    if do == "multipoles":
        ctx.legendre_project(case["nr"], case["ngauss"], case["npoly"], s["ar"], s["grids"], s["coef"])
        ctx.computePhil(s["ar"], s["coef"][0], *s["out"])
        return {"coef": s["coef"], "phil": s["out"][0], "Pr": s["out"][1], "Pr2": s["out"][2]}
    if do == "potential":
        ctx.potential_eval(s["pot"], s["Rz"], s["out"])
        return s["out"]
    if do == "actions":
        ctx.uvOrb_actions(s["pot"], s["delta"], s["pts"], s["out"])
        return s["out"]
    if do == "points":
        st = ctx.moments_points(s["pot"], s["delta"], s["df"], s["rule"], s["Rz"], s["out"])
        return {"out": s["out"], "bound": st.bound}
    if do == "iteration":
        st = ctx.computeNewPhi(s["pot"], s["delta"], s["df"], s["rule"], case["ngauss"], s["grids"], s["coef"],
                               *s["out"])
        return {"grids": s["grids"], "coef": s["coef"], "phil": s["out"][0], "Pr": s["out"][1], "Pr2": s["out"][2],
                "bound": st.bound, "failures": st.failures}
    if do == "los":
        st = ctx.los(s["pot"], s["delta"], s["df"], s["rule"], s["rhl_d"], KINDS[case["kind"]], s["Rzv"], s["out"])
        return {"out": s["out"], "bound": st.bound}
    if do == "batch":
        st = ctx.moments_batch(s["items"], s["rule"])
        return {"grids": [it[4] for it in s["items"]], "bound": st.bound, "failures": st.failures}
    if do == "surrogate":
        s["net"].moments(s["pot"], s["df"], s["rule"], case["ngauss"], s["grids"])
        return s["grids"]
    out = ctx.run_model(case["nr"], case["ngauss"], case["npoly"], 0.0, 0.0, s["df"], s["rule"],
                        itermax=case["iterations"], restart=s["tables"], delta_table=s["table"], keep_grids=True)
    return {k: out[k] for k in ("coef6", "phil", "Pr", "Pr2", "grids6", "bound", "failures", "iterations")}


def work(case):
    do = case["do"]
    if do == "batch":
        sizes = [(max(12, case["nr"] - 3 * i), max(3, case["ngauss"] - i)) for i in range(case["models"])]
        pts = sum(a * b for a, b in sizes)
        tab = sum(a * (1 + 3 * case["npoly"]) for a, _ in sizes)
        return {"bytes": 8.0 * (6 * pts + tab), "flops": FLOPS_PER_NODE * pts * case["nq"] ** 3}
    nr, npl, ng = case["nr"], case["npoly"], case.get("ngauss", 0)
    tab = nr * (1 + 3 * npl) + 60
    if do == "multipoles":
        return {"bytes": 8.0 * (nr + 6 * nr * ng + 9 * nr * npl), "flops": 12.0 * nr * ng * npl + 60.0 * nr * npl}
    if do == "potential":
        return {"bytes": 8.0 * (5 * case["n"] + tab), "flops": case["n"] * (40.0 + 40.0 * npl)}
    if do == "actions":
        return {"bytes": 8.0 * (7 * case["n"] + tab), "flops": FLOPS_PER_ORBIT * case["n"]}
    if do == "points":
        return {"bytes": 8.0 * (8 * case["n"] + tab), "flops": FLOPS_PER_NODE * case["n"] * case["nq"] ** 3}
    if do == "los":
        per = {"line": case["nq"] ** 3, "vphi": 22 * 22}.get(case["kind"], 22 * case["nq"])
        return {"bytes": 8.0 * (4 * case["n"] + tab), "flops": FLOPS_PER_NODE * case["n"] * per}
    nodes = nr * ng * case["nq"] ** 3
    if do == "surrogate":  # the layers 16-128-128-128-128-16 of the bound nodes
        return {"bytes": 8.0 * (6 * nr * ng + tab), "flops": 0.39 * nodes * 2 * (2 * 16 * 128 + 3 * 128 * 128)}
    it = case.get("iterations", 1)
    return {"bytes": 8.0 * (tab + 6 * nr * ng + 9 * nr * npl) * it, "flops": FLOPS_PER_NODE * nodes * it}


# ---------------------------------------------------- extended precision
def _exact_multipoles(s):
    case, ld = s["case"], np.longdouble
    nr, ng, npl = case["nr"], case["ngauss"], case["npoly"]
    ar, Q = s["ar"].cpu().numpy().astype(ld), s["grids"].cpu().numpy().astype(ld)
    c, w = np.polynomial.legendre.leggauss(ng)
    c, w = (c + 1) / 2, w / 2
    poly = np.array([2 * np.polynomial.legendre.Legendre.basis(2 * k)(c) * w for k in range(npl)]).astype(ld)
    order = np.argsort(-c) if F.gauleg(0.0, 1.0, ng)[0][0] > 0.5 else np.arange(ng)
    coef = np.einsum("kg,qng->qnk", poly[:, order], Q)
    coef[:, 0, :] = 0
    coef[1:, 0, 0] = 2 * Q[1:, 0, 0]
    coef[0, 0, 0] = 2 * ((Q[0, 2, 0] - Q[0, 1, 0]) / (ar[2] - ar[1]) * (ar[0] - ar[1]) + Q[0, 1, 0])
    phil, Pr, Pr2 = _solve(ar, coef[0])
    return {k: np.asarray(v, np.float64) for k, v in
            (("coef", coef), ("phil", phil), ("Pr", Pr), ("Pr2", Pr2))}


def _exact_potential(s):
    """Phi and its R and z derivatives by the tables' interpolation: linear in
    r with a quadratic correction in the ten innermost intervals, r^-(2k+1)
    beyond the grid, held inside ar[0]."""
    ld = np.longdouble
    ar, (T, TP, _) = s["ar"].astype(ld), [t.astype(ld) for t in s["tabs"]]
    R, z = s["Rz"].cpu().numpy().astype(ld).T
    nr, npl = T.shape
    r0 = np.sqrt(R * R + z * z)
    cp = z / r0
    r = np.maximum(r0, ar[0])
    sn, c = R / r, z / r
    ext = r >= ar[-1]
    b = np.clip(np.searchsorted(s["ar"], np.asarray(r, np.float64), side="right") - 1, 0, nr - 2)
    t = b + 1
    f1 = (r - ar[b]) / (ar[t] - ar[b])
    quad = (t < 10) & ~ext
    thr = np.where((f1 < 0.5) & (b > 0), b - 1, np.minimum(t + 1, nr - 1))
    f2 = (r - ar[t]) * (r - ar[b]) / np.where(quad, (ar[thr] - ar[t]) * (ar[thr] - ar[b]), ld(1))
    f3 = (ar[thr] - ar[b]) / (ar[t] - ar[b])
    x = np.where(ext, ar[-1] / r, ld(1))
    inside = lambda V: f1 * V[t] + (1 - f1) * V[b] + np.where(  # noqa: E731
        quad, f2 * (V[thr] - V[b] - f3 * (V[t] - V[b])), ld(0))
    phi, dr, dth = (np.zeros_like(r) for _ in range(3))
    for k in range(npl):
        basis = np.polynomial.legendre.Legendre.basis(2 * k)
        cf = basis.convert(kind=np.polynomial.Polynomial).coef.astype(ld)
        P = lambda u: np.polynomial.polynomial.polyval(u, cf)  # noqa: E731
        dP = np.polynomial.polynomial.polyval(c, np.polynomial.polynomial.polyder(cf)) if k else 0 * c
        out = T[-1, k] * x ** (2 * k + 1)
        ph = np.where(ext, out, inside(T[:, k]))
        dph = np.where(ext, -(2 * k + 1) * out / r, inside(TP[:, k]))
        phi, dr, dth = phi + ph * P(cp), dr + dph * P(c), dth + ph * dP
    dth = -np.sqrt(1 - c * c) * dth
    return np.stack([phi, dth * (c / r) + dr * sn, dth * (-sn / r) + dr * c], 1).astype(np.float64)


def exact(case, seed):
    """Closed forms of the multipole solve and the potential.  The other
    outputs are the reference algorithm's adaptive roots and quadratures, with
    its own tolerances, over up to millions of orbits: no closed form, and
    hours in extended precision."""
    if case["do"] == "multipoles":
        return _exact_multipoles(prepare(case, seed))
    if case["do"] == "potential":
        return _exact_potential(prepare(case, seed))
    return None

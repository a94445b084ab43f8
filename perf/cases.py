"""The timed workloads of the walker library: what a user has it do, through
the public entry points of ``rust_qmc_gb300``.

Every case names a kind of call, a system and its sizes:

  eval      System.eval_batch: psi, gradients, Laplacians and E_L of W
            configurations held on the host (one configuration is the trait
            call of a sampler that steps on the host)
  sampling  sr.sample_configurations: the configurations of one SR or geometry
            iteration, all-electron moves of a small ensemble
  vmc_all   vmc_run with all-electron moves: an energy of H2 or Li
  block     one block of a VMC run on resident walkers: single-electron sweeps,
            then the refresh and every walker's E_L
  dmc       IS-DMC steps of a resident population, E_ref fed back
  sr        System.logderiv_batch: log-derivatives, E_L, dE_L/dp and the SR sums
  forces    System.forces_batch: the Hellmann-Feynman forces and d ln|psi|/dR
  batch     steps of an uneven batch of systems, every set's E_L read back
"""
import math

import numpy as np

from rust_qmc_gb300 import _lib as L
from rust_qmc_gb300 import sr as SR
from rust_qmc_gb300 import systems as S
from rust_qmc_gb300.api import Batch, Context, System, Walkers, vmc_run

SPECS = {
    "h2": S.h2_mo,
    "li": S.lithium_atom,
    "ch4_min": S.methane_minimal,       # 9 AOs, seeded orthonormal MOs, 12 parameters
    "ch4_gto": S.methane_gto,           # 6-31G, 17 AOs
    "c6h6": S.benzene_minimal,          # 42 electrons, 36 AOs
    "c6h6_gto": S.benzene_gto,          # 6-31G, 66 AOs
    "heg": S.electron_gas,              # 54 electrons, Ewald
}
PREC = {"fp64": L.QMC_FP64, "fp32": L.QMC_FP32_REFINE}
MOVE = {"gauss": L.QMC_MOVE_ONE_GAUSS, "drift": L.QMC_MOVE_ONE_DRIFT, "all": L.QMC_MOVE_ALL_GAUSS,
        "box": L.QMC_MOVE_ALL_BOX}
BATCH_KINDS = ("h2", "li", "ch4_min", "c6h6", "heg")


def listed():
    return [
        # one configuration at a time: EnergyCalculator::local_energy as a host sampler calls it
        dict(name="eval_ch4_1", kind="eval", system="ch4_gto", W=1),
        # a set of benzene configurations from a file: psi, drift and E_L of each
        dict(name="eval_c6h6_500", kind="eval", system="c6h6", W=500),
        # one iteration's samples of the SR and geometry drivers at their default 20 walkers
        dict(name="sampling_ch4_20", kind="sampling", system="ch4_min", W=20, samples=1000, equil=100),
        # the reference's conf/h2.yaml run: 4096 walkers, box moves, 500 + 2000 steps
        dict(name="vmc_h2_4096", kind="vmc_all", system="h2", W=4096, move="box", step=1.0, burnin=500, steps=2000),
        # the 65 536-walker CH4 workload: 64 sweeps per refresh, FP32 walkers
        dict(name="block_ch4_65536", kind="block", system="ch4_min", W=65536, precision="fp32", move="gauss",
             step=0.3, sweeps=64),
        # MethaneGTO with the reference's own sampler (Langevin proposals) in FP64, an odd ensemble
        dict(name="block_ch4_drift_3001", kind="block", system="ch4_gto", W=3001, precision="fp64", move="drift",
             step=0.02, sweeps=10),
        # the benzene VMC workload: 16 384 walkers
        dict(name="block_c6h6_16384", kind="block", system="c6h6", W=16384, precision="fp32", move="gauss", step=0.3,
             sweeps=64),
        # one twist of an electron-gas run: E_L every 16 sweeps
        dict(name="block_heg_8192", kind="block", system="heg", W=8192, precision="fp32", move="gauss", step=2.0,
             sweeps=16),
        # the benzene IS-DMC workload at a smaller target population
        dict(name="dmc_c6h6_8192", kind="dmc", system="c6h6", W=8192, precision="fp32", tau=0.005, steps=4),
        # the gradient evaluation of an SR iteration over the default 5000 samples
        dict(name="sr_ch4_5000", kind="sr", system="ch4_min", W=5000),
        # the force evaluation of a geometry step over as many samples
        dict(name="forces_ch4_5000", kind="forces", system="ch4_gto", W=5000),
        # a parameter or twist scan: an uneven mix of small walker sets advanced together
        dict(name="batch_40", kind="batch", n=40, W_lo=256, W_hi=4096, sweeps=8, steps=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "sampling", "vmc_all", "block", "block", "block", "dmc", "sr", "forces", "batch"])
    if kind == "eval":
        system = rng.choice(["h2", "li", "ch4_min", "ch4_gto", "c6h6", "c6h6_gto", "heg"])
        return dict(kind=kind, system=system, W=_log_int(rng, 1, 500))
    if kind == "sampling":
        W = _log_int(rng, 8, 200)
        return dict(kind=kind, system=rng.choice(["h2", "li", "ch4_min", "ch4_gto"]), W=W,
                    samples=W * rng.randint(10, 40), equil=rng.randint(40, 100))
    if kind == "vmc_all":
        if rng.random() < 0.5:
            return dict(kind=kind, system="h2", W=_log_int(rng, 500, 16384), move="box", step=1.0,
                        burnin=rng.randint(50, 300), steps=rng.randint(200, 700))
        return dict(kind=kind, system="li", W=_log_int(rng, 500, 32768), move="all", step=1.0,
                    burnin=rng.randint(10, 50), steps=rng.randint(50, 150))
    if kind == "block":
        system = rng.choice(["li", "ch4_min", "ch4_gto", "c6h6", "c6h6_gto", "heg"])
        if system in ("li", "ch4_min", "ch4_gto") and rng.random() < 0.4:
            return dict(kind=kind, system=system, W=_log_int(rng, 64, 4000), precision="fp64",
                        move=rng.choice(["gauss", "drift"]), step=0.02 if system != "li" else 0.05,
                        sweeps=rng.randint(2, 10))
        hi = {"li": 65536, "ch4_min": 65536, "ch4_gto": 65536, "c6h6": 16384, "c6h6_gto": 8192, "heg": 8192}[system]
        return dict(kind=kind, system=system, W=_log_int(rng, hi // 64, hi), precision="fp32", move="gauss",
                    step=2.0 if system == "heg" else 0.3, sweeps=16 if system == "heg" else rng.choice([16, 32, 64]))
    if kind == "dmc":
        if rng.random() < 0.5:
            return dict(kind=kind, system="h2", W=_log_int(rng, 256, 16384), precision="fp64", tau=0.005,
                        steps=rng.randint(4, 20))
        return dict(kind=kind, system="c6h6", W=_log_int(rng, 256, 8192), precision="fp32", tau=0.005,
                    steps=rng.randint(2, 4))
    if kind == "sr":
        system = rng.choice(["ch4_min", "ch4_gto", "c6h6"])
        return dict(kind=kind, system=system, W=_log_int(rng, 200, 600 if system == "c6h6" else 20000))
    if kind == "forces":
        system = rng.choice(["h2", "ch4_min", "ch4_gto"])
        return dict(kind=kind, system=system, W=_log_int(rng, 100, 10000))
    return dict(kind=kind, n=rng.randint(8, 40), W_lo=256, W_hi=_log_int(rng, 300, 4096), sweeps=rng.choice([2, 4, 8]),
                steps=1)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_CTX = None


def _ctx():
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
    return _CTX


def _configurations(spec, W, seed):
    """W configurations near |psi|^2: electrons around their starting nuclei
    with a hydrogen-like radial density, uniform in a periodic box."""
    rng = np.random.default_rng([seed, 17])
    N = spec.n_elec
    if spec.box_L > 0:
        return rng.uniform(0.0, spec.box_L, size=(W, N, 3))
    nuc = np.where(spec.init_nuc < 0, 0, spec.init_nuc)
    # the first two electrons of a heavy nucleus feel its core, the others a valence shell
    zeta = np.ones(N)
    seen = {}
    for e, I in enumerate(nuc):
        k = seen[I] = seen.get(I, 0) + 1
        Z = spec.nuc_charge[I]
        zeta[e] = Z - 0.3 if (k <= 2 and Z > 2) else (1.2 if Z <= 2 else max(0.65, 0.5 * (Z - 2.8)))
    r = rng.gamma(3.0, 1.0, size=(W, N)) / (2.0 * zeta)
    v = rng.standard_normal((W, N, 3))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    return spec.nuc_pos[nuc][None] + r[..., None] * v


def _small_seed(seed):
    return 1 + seed % 1000003


def prepare(case, seed):
    kind = case["kind"]
    seed = _small_seed(seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    spec = SPECS[case["system"]]()
    st = dict(case=case, seed=seed, sys=System(_ctx(), spec))
    if kind in ("eval", "sr", "forces"):
        st["pos"] = _configurations(spec, case["W"], seed)
    elif kind == "block":
        wk = Walkers(st["sys"], case["W"], PREC[case["precision"]])
        wk.init(seed)
        wk.refresh()
        for k in range(2):
            wk.sweep(MOVE["gauss"], 8, 8 * k, seed=seed, step=case["step"] if case["move"] == "gauss" else 0.3,
                     count=False)
            wk.refresh()
        st.update(wk=wk, step0=16)
    elif kind == "dmc":
        wk = Walkers(st["sys"], case["W"], PREC[case["precision"]], capacity=4 * case["W"])
        wk.init(seed)
        wk.refresh()
        for k in range(4):
            wk.sweep(MOVE["gauss"], 32, 32 * k, seed=seed, step=0.3, count=False)
            e_ref = wk.refresh() / wk.W
        st.update(wk=wk, step0=0, e_ref=e_ref)
    return st


def _prepare_batch(case, seed):
    rng = np.random.default_rng([case["n"], case["W_lo"], case["W_hi"]])
    kinds = [BATCH_KINDS[i % len(BATCH_KINDS)] for i in range(case["n"])]
    sizes = [int(w) for w in rng.integers(case["W_lo"], case["W_hi"] + 1, size=case["n"])]
    systems = {k: System(_ctx(), SPECS[k]()) for k in sorted(set(kinds))}
    sets = []
    for i, (k, W) in enumerate(zip(kinds, sizes)):
        wk = Walkers(systems[k], W, PREC["fp32"])
        wk.init(seed + i)
        wk.refresh()
        sets.append(wk)
    return dict(case=case, seed=seed, systems=systems, sets=sets, batch=Batch(_ctx(), sets), step0=0)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "eval":
        return st["sys"].eval_batch(st["pos"], L.QMC_FP64)
    if kind == "sampling":
        return SR.sample_configurations(st["sys"], case["W"], case["samples"], case["equil"], 0.5, st["seed"])
    if kind == "vmc_all":
        return vmc_run(st["sys"], n_walkers=case["W"], n_steps=case["steps"], n_burnin=case["burnin"],
                       move_kind=MOVE[case["move"]], step=case["step"], precision=L.QMC_FP64, seed=st["seed"])
    if kind == "block":
        wk = st["wk"]
        accepted = wk.sweep(MOVE[case["move"]], case["sweeps"], st["step0"], seed=st["seed"], step=case["step"],
                            tau=case["step"])
        st["step0"] += case["sweeps"]
        e_sum = wk.refresh()
        return (accepted, e_sum) + wk.state()
    if kind == "dmc":
        wk, tau = st["wk"], case["tau"]
        out = []
        for _ in range(case["steps"]):
            n, em = wk.dmc_step(tau, st["e_ref"], seed=st["seed"], step=st["step0"], fp64_measure=True,
                                branch_cut=2.0 / math.sqrt(tau))
            st["step0"] += 1
            st["e_ref"] = em - 0.5 * math.log(n / case["W"]) / tau
            out.append((n, em))
        return out
    if kind == "sr":
        return st["sys"].logderiv_batch(st["pos"], sums=True, el_derivs=True)
    if kind == "forces":
        return st["sys"].forces_batch(st["pos"])
    e = st["batch"].run_steps(MOVE["gauss"], case["steps"], case["sweeps"], st["step0"], st["seed"], step=0.3)
    st["step0"] += case["steps"] * case["sweeps"]
    return e, np.concatenate([w.state()[2] for w in st["sets"]])


# ---------------------------------------------------------------------------
# Bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(name):
    """(electrons, state scalars of a walker, operations of one evaluation
    with E_L, operations of one single-electron proposal)."""
    spec = SPECS[name]()
    N = spec.n_elec
    up = int((spec.spins > 0).sum())
    sectors = (up, N - up)
    if spec.box_L > 0:
        dets = sum(8 * n ** 3 + 40 * n * n for n in sectors)
        nk = 462                                        # reciprocal vectors of the default splitting
        ev = dets + 40 * N * (N - 1) // 2 + 8 * N * nk
        return N, 3 * N + 4 * sum(n * n for n in sectors) // 2, ev, 30 * up + 16 * up * up // 2 + 40 * N
    n_prim = len(spec.prim_exp)
    n_ao = len(spec.ao_nuc)
    dets = sum(2 * n ** 3 for n in sectors)
    pairs = N * (N - 1) // 2 + N * spec.n_nuc
    occ = max(sectors)
    ev = N * (10 * n_prim + 10 * n_ao + 2 * n_ao * occ + 10 * n_ao) + dets + 40 * pairs
    mv = 4 * n_prim + 2 * n_ao * occ + 2 * occ * occ + 15 * (N + spec.n_nuc)
    return N, 3 * N + sum(n * n for n in sectors), ev, mv


def work(case):
    kind = case["kind"]
    if kind == "batch":
        W = case["n"] * (case["W_lo"] + case["W_hi"]) / 2.0 / len(BATCH_KINDS)
        b = f = 0.0
        for k in BATCH_KINDS:
            N, state, ev, mv = _counts(k)
            b += W * case["steps"] * (2 * 4 * state + 8)
            f += W * case["steps"] * (case["sweeps"] * N * mv + ev)
        return dict(bytes=b, flops=f)
    N, state, ev, mv = _counts(case["system"])
    W = case["W"]
    if kind == "eval":
        return dict(bytes=W * 8.0 * (3 * N + 4 * N + 2) + 4.0 * W, flops=float(W) * ev)
    if kind == "sampling":
        rounds = max(1, case["samples"] // W)
        steps = case["equil"] + 5 * rounds
        return dict(bytes=rounds * W * N * 24.0, flops=float(W) * steps * ev)
    if kind == "vmc_all":
        return dict(bytes=W * N * 24.0 + 8.0 * case["steps"], flops=float(W) * (case["burnin"] + case["steps"]) * ev)
    if kind == "block":
        size = 4 if case["precision"] == "fp32" else 8
        return dict(bytes=W * (2.0 * size * state + 20), flops=float(W) * (case["sweeps"] * N * mv + ev))
    if kind == "dmc":
        size = 4 if case["precision"] == "fp32" else 8
        return dict(bytes=case["steps"] * W * (2.0 * size * state + 16), flops=float(W) * case["steps"] * (N * 2 * mv + ev))
    spec = SPECS[case["system"]]()
    if kind == "sr":
        P = spec.n_params
        return dict(bytes=W * 8.0 * (3 * N + 2 * P + 1), flops=float(W) * (ev + P * (P + 10 * N)))
    return dict(bytes=W * 8.0 * (3 * N + 6 * spec.n_nuc), flops=float(W) * (ev + 20 * N * spec.n_nuc))


# ---------------------------------------------------------------------------
# The same quantities in plain numpy, 64 bits
# ---------------------------------------------------------------------------
def _aos(spec, r):
    """Values, gradients and Laplacians of the AOs at points r [..., 3]."""
    n = len(spec.ao_nuc)
    v = np.zeros(r.shape[:-1] + (n,))
    g = np.zeros(r.shape[:-1] + (n, 3))
    lap = np.zeros_like(v)
    for a in range(n):
        d = r - spec.nuc_pos[spec.ao_nuc[a]]
        r2 = (d * d).sum(-1)
        p = slice(spec.ao_prim_off[a], spec.ao_prim_off[a + 1])
        ex, co, pw = spec.prim_exp[p], spec.prim_coef[p], spec.prim_pow[p]
        if spec.basis_kind == L.QMC_BASIS_GTO:
            e = co * np.exp(-ex * r2[..., None])
            R0, R1, R2 = e.sum(-1), (ex * e).sum(-1), (ex * ex * e).sum(-1)
            if spec.ao_l[a] == 0:
                v[..., a] = R0
                g[..., a, :] = -2 * R1[..., None] * d
                lap[..., a] = -6 * R1 + 4 * r2 * R2
            else:
                m = spec.ao_m[a]
                x = d[..., m]
                v[..., a] = x * R0
                g[..., a, :] = -2 * (x * R1)[..., None] * d
                g[..., a, m] += R0
                lap[..., a] = x * (-10 * R1 + 4 * r2 * R2)
        else:
            q = np.sqrt(r2)[..., None]
            e = np.exp(-ex * q)
            f0 = q ** pw * e
            n1 = np.where(pw > 0, pw * q ** np.maximum(pw - 1, 0), 0.0) * e
            n2 = np.where(pw > 1, pw * (pw - 1) * q ** np.maximum(pw - 2, 0), 0.0) * e
            f1 = n1 - ex * f0
            f2 = n2 - 2 * ex * n1 + ex * ex * f0
            q = q[..., 0]
            v[..., a] = (co * f0).sum(-1)
            g[..., a, :] = ((co * f1).sum(-1) / q)[..., None] * d
            lap[..., a] = (co * f2).sum(-1) + 2 * (co * f1).sum(-1) / q
    return v, g, lap


def _pair_u(spec, r, para):
    """u, u'/r, u'' + 2 u'/r of the electron pairs at distances r."""
    if spec.jastrow_kind == L.QMC_JAS_PADE_F:
        inv = 1.0 / (1.0 + r / spec.jas_F)
        return -0.5 * spec.jas_F * inv, 0.5 * inv ** 2 / r, inv ** 3 / r
    k = 1 if para else 0
    if spec.jastrow_kind == L.QMC_JAS_PADE_EEN:
        return _pade(spec.jas[2 + k], spec.jas[k], r)
    a, b, c = spec.jas[2 + k], 1.0 / spec.jas_F, 0.2 / spec.jas_F ** 2
    den = 1.0 + b * r + c * r * r
    u, d1 = a * r / den, a * (1.0 - c * r * r) / den ** 2
    d2 = -2.0 * a * (c * r * den + (1.0 - c * r * r) * (b + 2.0 * c * r)) / den ** 3
    on = r < 0.5 * spec.box_L
    return np.where(on, u, 0.0), np.where(on, d1 / r, 0.0), np.where(on, d2 + 2.0 * d1 / r, 0.0)


def _pade(a, b, r):
    inv = 1.0 / (1.0 + b * r)
    return a * r * inv, a * inv ** 2 / r, 2 * a * inv ** 2 / r - 2 * a * b * inv ** 3


def _evaluate(spec, pos):
    """log|psi|, grad ln psi, lap psi / psi and E_L, with the pieces the
    derivatives need."""
    W, N = pos.shape[:2]
    up = spec.spins > 0
    order = [np.nonzero(up)[0], np.nonzero(~up)[0]]
    logabs = np.zeros(W)
    gd = np.zeros((W, N, 3))
    ld = np.zeros((W, N))
    sectors = []
    if spec.box_L > 0:
        for el in order:
            k = spec.mo_coef[spec.occ[el]]
            D = np.exp(1j * (pos[:, el] @ k.T))
            B = np.linalg.inv(D)
            logabs += np.linalg.slogdet(D)[1]
            w = D * B.transpose(0, 2, 1)
            gd[:, el] = np.real(1j * (w @ k))
            ld[:, el] = -np.real(w @ (k * k).sum(1))
    else:
        v, g, lap = _aos(spec, pos)
        for el in order:
            if not len(el):
                continue
            C = spec.mo_coef[spec.occ[el]].T
            D = v[:, el] @ C
            B = np.linalg.inv(D)
            logabs += np.linalg.slogdet(D)[1]
            cB = np.einsum("ak,wkq->wqa", C, B)
            gd[:, el] = np.einsum("wqa,wqac->wqc", cB, g[:, el])
            ld[:, el] = np.einsum("wqa,wqa->wq", cB, lap[:, el])
            sectors.append((el, cB, B))
    gj = np.zeros((W, N, 3))
    lj = np.zeros((W, N))
    sq = np.zeros((W, N))
    u = np.zeros(W)
    V = np.full(W, spec.v_nn())
    for i in range(N):
        for j in range(i + 1, N):
            d = pos[:, i] - pos[:, j]
            if spec.box_L > 0:
                d = d - spec.box_L * np.rint(d / spec.box_L)
            r = np.sqrt((d * d).sum(1))
            if spec.box_L == 0:
                V += 1.0 / r
            uu, f, t = _pair_u(spec, r, up[i] == up[j])
            u += uu
            gj[:, i] += f[:, None] * d
            gj[:, j] -= f[:, None] * d
            for e in (i, j):
                lj[:, e] += t
                sq[:, e] += (f * r) ** 2
        for I in range(spec.n_nuc):
            d = pos[:, i] - spec.nuc_pos[I]
            r = np.sqrt((d * d).sum(1))
            V -= spec.nuc_charge[I] / r
            if spec.jastrow_kind == L.QMC_JAS_PADE_EEN:
                s = spec.nuc_species[I]
                uu, f, t = _pade(spec.jas[6 + s] * spec.nuc_charge[I], spec.jas[4 + s], r)
                u -= uu
                gj[:, i] -= f[:, None] * d
                lj[:, i] -= t
    if spec.box_L > 0:
        V += _ewald(spec, pos)
    qa = spec.jas_F if spec.quirks & L.QMC_QUIRK_J2_GRAD else 1.0
    extra = sq if spec.quirks & L.QMC_QUIRK_J2_LAP else (gj * gj).sum(2)
    lap = ld + 2 * qa * (gd * gj).sum(2) + lj + extra
    return dict(logabs=logabs + u, grad=gd + qa * gj, lap=lap, e_local=V - 0.5 * lap.sum(1), sectors=sectors)


def _ewald(spec, pos):
    """One-component-plasma Ewald energy with the description's splitting."""
    from math import erfc, pi, sqrt
    box, N = spec.box_L, spec.n_elec
    vol, al, K = box ** 3, spec.jas[4] / box, int(spec.jas[5])
    ferfc = np.vectorize(erfc)
    V = np.zeros(len(pos))
    cells = [np.array([a, b, c]) * box for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    iu = np.triu_indices(N, 1)
    d = pos[:, iu[0]] - pos[:, iu[1]]
    d -= box * np.rint(d / box)
    for cell in cells:
        r = np.sqrt(((d + cell) ** 2).sum(2))
        near = r < 5.6 / al
        t = np.zeros_like(r)
        t[near] = ferfc(al * r[near]) / r[near]
        V += t.sum(1)
    n = np.array([(a, b, c) for a in range(K + 1) for b in range(-K, K + 1) for c in range(-K, K + 1)
                  if (a, b, c) > (0, 0, 0) and a * a + b * b + c * c <= K * K])
    k = 2 * pi / box * n
    k2 = (k * k).sum(1)
    rho = np.exp(1j * (pos @ k.T)).sum(1)
    V += (np.abs(rho) ** 2) @ (4 * pi / vol * np.exp(-k2 / (4 * al * al)) / k2)
    img = sum(erfc(al * box * sqrt(a * a + b * b + c * c)) / (box * sqrt(a * a + b * b + c * c))
              for a in range(-3, 4) for b in range(-3, 4) for c in range(-3, 4) if a or b or c)
    return V + N * (0.5 * img - al / sqrt(pi) - pi * N / (2 * vol * al * al))


def _log_derivatives(spec, pos, ev):
    W, N = pos.shape[:2]
    O = np.zeros((W, spec.n_params))
    up = spec.spins > 0
    for i in range(N):
        for j in range(i + 1, N):
            c = 1 if up[i] == up[j] else 0
            r = np.sqrt(((pos[:, i] - pos[:, j]) ** 2).sum(1))
            inv = 1.0 / (1.0 + spec.jas[c] * r)
            O[:, c] -= spec.jas[2 + c] * (r * inv) ** 2
            O[:, 2 + c] += r * inv
        for I in range(spec.n_nuc):
            s, Z = spec.nuc_species[I], spec.nuc_charge[I]
            r = np.sqrt(((pos[:, i] - spec.nuc_pos[I]) ** 2).sum(1))
            inv = 1.0 / (1.0 + spec.jas[4 + s] * r)
            O[:, 4 + s] += spec.jas[6 + s] * Z * (r * inv) ** 2
            O[:, 6 + s] -= Z * r * inv
    if len(spec.rot_occ):
        v = _aos(spec, pos)[0]
        for q, (k, m) in enumerate(zip(spec.rot_occ, spec.rot_virt)):
            for el, _, B in ev["sectors"]:
                for c in np.nonzero(spec.occ[el] == k)[0]:
                    O[:, 8 + q] += (B[:, c] * (v[:, el] @ spec.mo_coef[m])).sum(1)
    return O


def _forces(spec, pos, ev):
    W, N = pos.shape[:2]
    F = np.zeros((W, spec.n_nuc, 3))
    om = np.zeros((W, spec.n_nuc, 3))
    g = _aos(spec, pos)[1]
    for I in range(spec.n_nuc):
        d = pos - spec.nuc_pos[I]
        r = np.sqrt((d * d).sum(2))[..., None]
        F[:, I] = (spec.nuc_charge[I] * d / r ** 3).sum(1)
        for J in range(spec.n_nuc):
            if J != I:
                x = spec.nuc_pos[I] - spec.nuc_pos[J]
                F[:, I] -= spec.nuc_charge[I] * spec.nuc_charge[J] * x / np.linalg.norm(x) ** 3
        on = spec.ao_nuc == I
        for el, cB, _ in ev["sectors"]:
            om[:, I] -= np.einsum("wqa,wqac->wc", cB[:, :, on], g[:, el][:, :, on])
        if spec.jastrow_kind == L.QMC_JAS_PADE_EEN:
            s = spec.nuc_species[I]
            f = _pade(spec.jas[6 + s] * spec.nuc_charge[I], spec.jas[4 + s], r)[1]
            om[:, I] += (f * d).sum(1)
    return F, om


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("eval", "sr", "forces"):
        return None
    spec = SPECS[case["system"]]()
    pos = _configurations(spec, case["W"], _small_seed(seed))
    ev = _evaluate(spec, pos)
    if kind == "eval":
        return dict(logabs=ev["logabs"], sign=None, grad=ev["grad"], lap=ev["lap"], e_local=ev["e_local"])
    if kind == "forces":
        return _forces(spec, pos, ev)
    O, E = _log_derivatives(spec, pos, ev), ev["e_local"]
    Om, Em = O.mean(0), E.mean()
    return O, E, None, O.T @ O / len(E) - np.outer(Om, Om), E @ O / len(E) - Em * Om, float(Em)

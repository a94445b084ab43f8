"""The warp-per-walker kernels (benzene, electron gas) and the DMC and SR reductions
at the sizes where their launches change: one walker, partial blocks of the sweep
(4 walkers), of the float-float refresh (12) and of the FP64 evaluation (4), bases
whose shells do not deal evenly into thirds, reciprocal cutoffs other than the
default.

Tolerances.  FP64 evaluation: 1e-9 of the norm over the set, as for every FP64
evaluation of the library.  E_L of a float-float refresh: 1e-6 Ha at the walkers' own
(FP32) positions.  FP32 chains: proposals carry a few roundings of coordinates below
16, 1e-4 with room; a ratio's relative error is FP32's 6e-8 times the conditioning of a
21 x 21 inverse after many updates, about 1e-4 and 2e-3 with room for |ratio|^2, so a
walker whose chain came that near to another decision may leave the oracle's, and one
walker in 16 may for worse conditioning."""
import copy

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu


def unshared_benzene():
    """Benzene whose nuclei differ in their shells: two carbons' p exponents are no
    longer their 2s shell's, so sp shells, lone s groups and lone p triplets all occur,
    in numbers that three does not divide."""
    spec = Q.benzene_minimal()
    exps = np.array(spec.prim_exp, dtype=float)
    for a in range(len(spec.ao_nuc)):
        if spec.ao_l[a] == 1 and spec.ao_nuc[a] in (1, 4):
            exps[spec.ao_prim_off[a]:spec.ao_prim_off[a + 1]] *= 1.1
    spec = copy.copy(spec)
    spec.prim_exp = exps
    return spec


BENZENES = {"min": Q.benzene_minimal, "gto": Q.benzene_gto, "unshared": unshared_benzene}


def _close(a, b, tol=1e-9):
    assert np.linalg.norm(np.asarray(a) - b) <= tol * np.linalg.norm(b)


def _same_chain(got, want, margin, box=0.0):
    d = got - want
    if box:
        d -= box * np.rint(d / box)
    off = ~np.all(np.abs(d) < 1e-4, axis=(1, 2)) & (margin > 2e-3)
    assert off.sum() <= len(off) // 16, margin[off]


@pytest.mark.parametrize("name, W", [("min", 1), ("min", 3), ("min", 5), ("gto", 4), ("unshared", 6)])
def test_benzene_evaluation(ctx, oracle, name, W):
    spec = BENZENES[name]()
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, W, seed=30 + W)
    got, want = sysh.eval_batch(pos), oracle.evaluate(spec, pos)
    assert np.array_equal(got["sign"], want["sign"])
    for k in ("logabs", "grad", "lap", "e_local"):
        _close(got[k], want[k])
    sysh.close()


@pytest.mark.parametrize("prec", [L.QMC_FP32_REFINE, L.QMC_FP64])
@pytest.mark.parametrize("name, W", [("min", 1), ("min", 11), ("min", 12), ("min", 13), ("gto", 5), ("unshared", 14)])
def test_benzene_refresh(ctx, oracle, name, W, prec):
    """Standalone and as one class of a batch."""
    spec = BENZENES[name]()
    sysh = Q.System(ctx, spec)
    sets = [Q.Walkers(sysh, W, prec) for _ in range(2)]
    for wk in sets:
        wk.init(seed=9)
        wk.refresh()
        wk.sweep(L.QMC_MOVE_ONE_GAUSS, 4, 0, seed=10, step=0.3)
    sets[0].refresh()
    batch = Q.Batch(ctx, sets[1:])
    mean = batch.refresh()
    want = oracle.evaluate(spec, sets[0].get_positions())
    for wk in sets:
        la, sg, el = wk.state()
        assert np.max(np.abs(el - want["e_local"])) <= 1e-6
        assert np.max(np.abs(la - want["logabs"])) <= 1e-6 and np.array_equal(sg, want["sign"])
    assert abs(mean[0] - want["e_local"].mean()) <= 1e-6
    batch.close()
    for wk in sets:
        wk.close()
    sysh.close()


@pytest.mark.parametrize("move", [L.QMC_MOVE_ONE_GAUSS, L.QMC_MOVE_ONE_DRIFT])
@pytest.mark.parametrize("name, W", [("min", 1), ("min", 33), ("gto", 6), ("unshared", 18)])
def test_benzene_fp32_chain(ctx, oracle, name, W, move):
    spec = BENZENES[name]()
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP32_REFINE)
    wk.init(seed=5)
    wk.refresh()
    pos0 = wk.get_positions()
    kw = dict(step=0.3, tau=0.005, max_drift=1.0)
    wk.sweep(move, 2, 3, seed=606, **kw)
    want, _, _, margin = oracle.sweeps(spec, pos0, 2, 3, move, 606, want_energy=False, want_margin=True, **kw)
    _same_chain(wk.get_positions(), want, margin)
    wk.close()
    sysh.close()


@pytest.mark.parametrize("kmax", [1, 3, 9])
@pytest.mark.parametrize("prec", [L.QMC_FP32_REFINE, L.QMC_FP64])
def test_electron_gas_reciprocal_cutoff(ctx, oracle, kmax, prec):
    spec = Q.electron_gas(kmax=kmax)
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, 5, prec)
    wk.init(seed=17)
    wk.refresh()
    want = oracle.evaluate(spec, wk.get_positions())
    assert np.max(np.abs(wk.state()[2] - want["e_local"])) <= 1e-6
    wk.close()
    sysh.close()


def test_electron_gas_batch_follows_a_larger_cutoff(ctx):
    """A batch captured at one reciprocal cutoff, its system then set to a larger one."""
    sysh = Q.System(ctx, Q.electron_gas(kmax=3))
    a, b = (Q.Walkers(sysh, 6, L.QMC_FP32_REFINE) for _ in range(2))
    for wk in (a, b):
        wk.init(seed=2)
        wk.refresh()
    batch = Q.Batch(ctx, [a])
    batch.run_steps(L.QMC_MOVE_ONE_GAUSS, 1, 1, 0, 7, step=1.0)
    b.sweep(L.QMC_MOVE_ONE_GAUSS, 1, 0, seed=Q.batch_system_seed(7, 0), step=1.0)
    p = sysh.get_params()
    p[5] = 8
    sysh.set_params(p)
    series = batch.run_steps(L.QMC_MOVE_ONE_GAUSS, 1, 1, 1, 7, step=1.0)
    b.sweep(L.QMC_MOVE_ONE_GAUSS, 1, 1, seed=Q.batch_system_seed(7, 0), step=1.0)
    b.refresh()
    assert np.array_equal(a.state()[2], b.state()[2])
    np.testing.assert_allclose(np.ravel(series), b.state()[2].mean(), rtol=1e-12, atol=0)
    batch.close()
    a.close()
    b.close()
    sysh.close()


@pytest.mark.parametrize("form", ["rpa", "pade", "yukawa"])
@pytest.mark.parametrize("W", [1, 18])
def test_electron_gas_fp32_chain(ctx, oracle, form, W):
    spec = Q.electron_gas(form=form)
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP32_REFINE)
    wk.init(seed=15)
    wk.refresh()
    pos0 = wk.get_positions()
    wk.sweep(L.QMC_MOVE_ONE_GAUSS, 2, 2, seed=616, step=1.0)
    want, _, _, margin = oracle.sweeps(spec, pos0, 2, 2, L.QMC_MOVE_ONE_GAUSS, 616, step=1.0, want_energy=False,
                                       want_margin=True)
    _same_chain(wk.get_positions(), want, margin, spec.box_L)
    wk.close()
    sysh.close()


@pytest.mark.parametrize("W", [1, 255, 256, 257, 1025])
def test_dmc_compaction(ctx, oracle, W):
    """Branching counts, their scan and the gather across block edges: populations and
    mean energies of three steps against the oracle's."""
    spec = Q.h2_mo()
    sysh = Q.System(ctx, spec)
    tau, seed = 0.02, 13
    wk = Q.Walkers(sysh, W, L.QMC_FP64, capacity=4 * W + 8)
    wk.init(seed=12)
    e_ref = wk.refresh() / W
    pos0 = wk.get_positions()
    pops, means, er = [], [], e_ref
    for t in range(3):
        n, em = wk.dmc_step(tau, er, seed=seed, step=t)
        pops.append(n)
        means.append(em)
        if n == 0:
            break
        er = em - 0.5 * np.log(n / W) / tau
    _, pops_o, means_o, _ = oracle.dmc(spec, pos0, len(pops), tau, e_ref, W, seed, fixed_node=True)
    assert list(pops) == list(pops_o)
    np.testing.assert_allclose(means, means_o, rtol=1e-9, atol=1e-9)
    wk.close()
    sysh.close()


@pytest.mark.parametrize("W", [1, 31, 32, 33, 97])
def test_sr_sums(ctx, W):
    """S, f and the mean energy from sums over chunks of 32 walkers, against numpy's
    from the same rows (64-bit sums of up to 97 terms: 1e-12 of the largest)."""
    spec = Q.methane_minimal()
    sysh = Q.System(ctx, spec)
    O, E, S, f, em = sysh.logderiv_batch(random_configs(spec, W, seed=W), sums=True)
    Om = O.mean(0)
    S2 = O.T @ O / W
    np.testing.assert_allclose(S, S2 - np.outer(Om, Om), rtol=0, atol=1e-12 * np.abs(S2).max())
    f2 = (E[:, None] * O).mean(0)
    np.testing.assert_allclose(f, f2 - E.mean() * Om, rtol=0, atol=1e-12 * np.abs(E).max() * np.abs(O).max())
    assert abs(em - E.mean()) <= 1e-12 * np.abs(E).max()
    sysh.close()


@pytest.mark.parametrize("W", [1, 3, 5])
def test_benzene_sr_rows(ctx, oracle, W):
    """A warp per configuration, partial blocks of four: O_p against the oracle, dE_L/dp
    against differences of E_L (step 1e-4 of a parameter: 1e-5 of the largest)."""
    spec = Q.benzene_gto(2.0, 3.0)
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, W, seed=40 + W)
    O, E, dE = sysh.logderiv_batch(pos, el_derivs=True)
    _close(O, oracle.log_derivatives(spec, pos))
    p, h = sysh.get_params(), 1e-4
    for k in range(len(p)):
        e = []
        for s in (h, -h):
            q = p.copy()
            q[k] += s
            sysh.set_params(q)
            e.append(sysh.eval_batch(pos)["e_local"])
        want = (e[0] - e[1]) / (2 * h)
        assert np.max(np.abs(dE[:, k] - want)) <= 1e-5 * max(1.0, np.max(np.abs(dE)))
    sysh.close()

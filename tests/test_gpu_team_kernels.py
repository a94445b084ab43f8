"""FP64 team kernels (a team of lanes per walker; H2, Li, CH4) at the sizes where
their launches change: one walker, partial blocks, and the ensemble size up to
which a block is a single warp (152 SMs x 4 sub-partitions of warps: 4864 H2,
2432 Li, 608 CH4 walkers).  Tolerances: FP64 evaluation with reciprocals to
1e-14, amplified by the conditioning of configurations near a node; 1e-9 of the
norm over the set, as for every FP64 evaluation of the library.  Trajectories
of Gaussian and box moves are sums of proposals, equal to rounding unless a
decision lies within rounding of its threshold."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu

SPECS = {"h2": Q.h2_mo, "li": lambda: Q.lithium_atom(reference_quirks=True), "ch4_gto": Q.methane_gto,
         "ch4_min": Q.methane_minimal}


def _close(a, b, tol=1e-9):
    assert np.linalg.norm(np.asarray(a) - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("W", [1, 3, 5, 33])
@pytest.mark.parametrize("name", sorted(SPECS))
def test_evaluation_matches_oracle(ctx, oracle, name, W):
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, W, seed=100 + W)
    got, want = sysh.eval_batch(pos), oracle.evaluate(spec, pos)
    assert np.array_equal(got["sign"], want["sign"])
    for k in ("logabs", "grad", "lap", "e_local"):
        _close(got[k], want[k])
    F, om = sysh.forces_batch(pos)
    Fo, omo = oracle.forces(spec, pos)[:2]
    _close(F, Fo)
    _close(om, omo)
    sysh.close()


@pytest.mark.parametrize("move", [L.QMC_MOVE_ALL_BOX, L.QMC_MOVE_ALL_GAUSS])
@pytest.mark.parametrize("name, W", [("h2", 1), ("h2", 4864), ("h2", 4865), ("li", 7), ("li", 2433), ("ch4_gto", 608),
                                     ("ch4_min", 20), ("ch4_min", 609)])
def test_steps_match_oracle(ctx, oracle, name, W, move):
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    pos = random_configs(spec, W, seed=7)
    wk.set_positions(pos)
    wk.refresh()
    n, step, seed = 3, 0.4, 99
    acc = wk.sweep(move, n, 5, seed=seed, step=step)
    want, acc_o, el_o = oracle.sweeps(spec, pos, n, 5, move, seed, step=step)
    got = wk.get_positions()
    same = np.all(np.abs(got - want) < 1e-9, axis=(1, 2))
    assert same.mean() >= 0.999, same.mean()
    if same.all():
        assert acc == acc_o.sum()
    _close(wk.state()[2][same], oracle.evaluate(spec, got)["e_local"][same])
    wk.close()
    sysh.close()


@pytest.mark.parametrize("name, W", [("h2", 37), ("h2", 4900), ("ch4_min", 5)])
@pytest.mark.parametrize("steps", [1, 32, 33])
def test_recorded_energies_are_the_steps_means(ctx, name, W, steps):
    """vmc_run's per-step means (recorded 32 steps at a time) against single steps."""
    sysh = Q.System(ctx, SPECS[name]())
    r = Q.vmc_run(sysh, n_walkers=W, n_steps=steps, n_burnin=2, move_kind=L.QMC_MOVE_ALL_GAUSS, step=0.4, seed=3)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    wk.init(seed=3)
    wk.refresh()
    wk.sweep(L.QMC_MOVE_ALL_GAUSS, 2, 0, seed=3, step=0.4)
    means = []
    for t in range(steps):
        wk.sweep(L.QMC_MOVE_ALL_GAUSS, 1, 2 + t, seed=3, step=0.4)
        means.append(wk.state()[2].mean())
    np.testing.assert_allclose(r["energies"], means, rtol=1e-11, atol=0)
    wk.close()
    sysh.close()


@pytest.mark.parametrize("move", [L.QMC_MOVE_ONE_GAUSS, L.QMC_MOVE_ONE_DRIFT])
@pytest.mark.parametrize("name, W", [("h2", 1), ("h2", 6144), ("h2", 6145), ("h2", 10240), ("h2", 10241), ("li", 9),
                                     ("ch4_gto", 5), ("ch4_min", 3), ("ch4_min", 130)])
def test_sweeps_match_oracle(ctx, oracle, name, W, move):
    """Single-electron sweeps on both sides of the size where a thread per walker
    takes over (6144 Gaussian, 10 240 Langevin), and with partly filled warps."""
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    pos = random_configs(spec, W, seed=11)
    wk.set_positions(pos)
    wk.refresh()
    n, seed = 3, 77
    acc = wk.sweep(move, n, 4, seed=seed, step=0.3, tau=0.02)
    want, acc_o, _ = oracle.sweeps(spec, pos, n, 4, move, seed, step=0.3, tau=0.02, want_energy=False)
    got = wk.get_positions()
    same = np.all(np.abs(got - want) < 1e-9, axis=(1, 2))
    assert same.mean() >= 0.98, same.mean()
    if same.all():
        assert acc == acc_o.sum()
    # the updated inverse gives the sign a rebuild gives
    s0 = wk.state()[1]
    wk.rebuild_inverse()
    assert np.array_equal(s0, wk.state()[1])
    assert wk.status() == 0
    wk.close()
    sysh.close()


@pytest.mark.parametrize("name, W", [("h2", 9216), ("h2", 9217), ("li", 9217), ("ch4_min", 9217)])
def test_refresh_and_recorded_steps_across_the_size_rule(ctx, oracle, name, W):
    """Refresh and recorded steps on both sides of 9216 walkers: E_L of the first
    and last walkers against the oracle, the recorded means against single steps."""
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    wk.init(seed=5)
    s, el = wk.refresh(want_energies=True)
    pick = np.r_[0:40, W - 40:W]
    _close(el[pick], oracle.evaluate(spec, wk.get_positions()[pick])["e_local"])
    np.testing.assert_allclose(s, el.sum(), rtol=1e-11)
    r = Q.vmc_run(sysh, n_walkers=W, n_steps=3, move_kind=L.QMC_MOVE_ALL_GAUSS, step=0.4, seed=5)
    means = []
    for t in range(3):
        wk.sweep(L.QMC_MOVE_ALL_GAUSS, 1, t, seed=5, step=0.4)
        means.append(wk.state()[2].mean())
    np.testing.assert_allclose(r["energies"], means, rtol=1e-9, atol=0)
    wk.close()
    sysh.close()


@pytest.mark.parametrize("name", ["ch4_gto", "ch4_min"])
def test_sr_rows_do_not_depend_on_the_batch(ctx, name):
    """Rows of a batch above the team kernels' size (9216) against the same
    configurations in a small batch: two FP64 routes, 1e-9 of the norm each as above."""
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, 9217, seed=3)
    big = sysh.logderiv_batch(pos, el_derivs=True)
    rows = np.r_[0:40, 9177:9217]
    small = sysh.logderiv_batch(pos[rows], el_derivs=True)
    for a, b in zip(big, small):
        a = np.asarray(a)[rows]
        for x, y in zip(a, b):
            _close(x, y, 1e-7)
        _close(a, b)
    sysh.close()

"""FP64 paths with negative Pade denominators 1 + b r: the parameters are any finite
numbers (the F of H2 and Li has to be positive).  b = -5 puts the pole at 0.2 bohr, so
nearly every pair lies beyond it.  Tolerances: an evaluation 1e-9 of the norm
over the set, as for every FP64 evaluation of the library; sweeps follow the
oracle's decisions unless one lies within rounding of its threshold."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu


def _spec(name):
    spec = {"ch4_gto": Q.methane_gto, "ch4_min": Q.methane_minimal, "c6h6": Q.benzene_minimal}[name]()
    p = spec.params()
    p[[0, 1, 4, 5]] = -5.0
    return spec.with_params(p)


@pytest.mark.parametrize("name, W", [("ch4_gto", 9), ("ch4_min", 9), ("c6h6", 5), ("ch4_min", 9217)])
def test_evaluation(ctx, oracle, name, W):
    spec = _spec(name)
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, W, seed=50 + W)
    got, want = sysh.eval_batch(pos), oracle.evaluate(spec, pos)
    assert np.array_equal(got["sign"], want["sign"])
    for k in ("logabs", "grad", "lap", "e_local"):
        assert np.linalg.norm(got[k] - want[k]) <= 1e-9 * np.linalg.norm(want[k]), k
    sysh.close()


@pytest.mark.parametrize("move", [L.QMC_MOVE_ALL_GAUSS, L.QMC_MOVE_ONE_GAUSS, L.QMC_MOVE_ONE_DRIFT])
@pytest.mark.parametrize("name, W", [("ch4_gto", 60), ("ch4_min", 100), ("ch4_min", 10241), ("c6h6", 8)])
def test_sweeps(ctx, oracle, name, W, move):
    if name == "c6h6" and move == L.QMC_MOVE_ALL_GAUSS:
        pytest.skip("not a move of benzene")
    spec = _spec(name)
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    pos = random_configs(spec, W, seed=3)
    wk.set_positions(pos)
    wk.refresh()
    wk.sweep(move, 2, 0, seed=9, step=0.3, tau=0.02)
    want = oracle.sweeps(spec, pos, 2, 0, move, 9, step=0.3, tau=0.02, want_energy=False)[0]
    same = np.all(np.abs(wk.get_positions() - want) < 1e-7, axis=(1, 2))
    assert same.mean() >= 0.95, same.mean()
    wk.close()
    sysh.close()

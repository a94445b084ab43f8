"""All-electron FP64 steps where the Jastrow exponent is hundreds (F = 1000: u near
-500 a pair, whose exponential alone is no double): accepted moves and positions against
the oracle, equal unless a decision lies within rounding of its threshold (log|psi| of
1500 carries 2e-13)."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu

SPECS = {"h2": lambda: Q.h2_mo(F=1000.0), "li": lambda: Q.lithium_atom(F=1000.0, reference_quirks=False)}


@pytest.mark.parametrize("move", [L.QMC_MOVE_ALL_GAUSS, L.QMC_MOVE_ALL_BOX])
@pytest.mark.parametrize("name", sorted(SPECS))
def test_steps_match_oracle(ctx, oracle, name, move):
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    W, n, step, seed = 300, 4, 0.4, 21
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    pos = random_configs(spec, W, seed=8)
    wk.set_positions(pos)
    wk.refresh()
    acc = wk.sweep(move, n, 0, seed=seed, step=step)
    want, acc_o, _ = oracle.sweeps(spec, pos, n, 0, move, seed, step=step)
    same = np.all(np.abs(wk.get_positions() - want) < 1e-9, axis=(1, 2))
    assert acc_o.sum() > 0 and same.mean() >= 0.999, (acc, same.mean())
    # recorded steps
    r = Q.vmc_run(sysh, n_walkers=W, n_steps=n, move_kind=move, step=step, seed=seed)
    assert r["acceptance_rate"] > 0
    wk.close()
    sysh.close()

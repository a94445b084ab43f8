"""FP64 walkers with a singular orbital matrix beside regular ones: an electron so far
out that its orbitals are zero.  Several H2 and Li walkers share a warp, so a singular one
must not hold up or change its neighbours; they match the oracle (1e-9 of the norm), and
the status says that there was one."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu

SINGULAR = 1                                       # first status bit


def _configs(name, W):
    """Configurations, every third singular; the same with regular ones in their places
    (the oracle does not step singular walkers)."""
    spec = {"h2": Q.h2_mo, "li": Q.lithium_atom, "ch4_min": Q.methane_minimal}[name]()
    regular = random_configs(spec, W, seed=2)
    pos = regular.copy()
    bad = np.zeros(W, bool)
    bad[1::3] = True
    pos[bad, 0] = [0.0, 0.0, 2000.0]
    return spec, pos, regular, bad


@pytest.mark.parametrize("name, W", [("h2", 2), ("h2", 40), ("li", 3), ("li", 40), ("ch4_min", 6)])
def test_neighbours_of_singular_walkers(ctx, oracle, name, W):
    spec, pos, regular, bad = _configs(name, W)
    sysh = Q.System(ctx, spec)
    got, want = sysh.eval_batch(pos), oracle.evaluate(spec, pos[~bad])
    assert np.array_equal(got["sign"][~bad], want["sign"])
    for k in ("logabs", "grad", "lap", "e_local"):
        assert np.linalg.norm(got[k][~bad] - want[k]) <= 1e-9 * np.linalg.norm(want[k]), k
    sysh.forces_batch(pos)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    for move in (L.QMC_MOVE_ALL_GAUSS, L.QMC_MOVE_ONE_GAUSS, L.QMC_MOVE_ONE_DRIFT):
        wk.set_positions(pos)
        wk.refresh()
        assert wk.status() & SINGULAR
        wk.sweep(move, 2, 0, seed=4, step=0.3, tau=0.02)
        after = oracle.sweeps(spec, regular, 2, 0, move, 4, step=0.3, tau=0.02, want_energy=False)[0]
        same = np.all(np.abs(wk.get_positions() - after) < 1e-7, axis=(1, 2))
        assert same[~bad].mean() >= 0.9
    wk.close()
    sysh.close()

"""SR rows with MO rotations: large batches go a thread per walker, smaller ones by
teams.  As in test_gpu_sr_large_batches only sums of 64-bit terms differ, and E_L is
measured against dE_L/dp; a rotation's terms are products with the inverse, an order of
magnitude above their sum next to a node: 1e-13.  O_p also against the oracle."""
import copy

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu


def _table_driven():
    """The 9-function CH4 without its last hydrogen's third primitive: a layout that is
    not compiled."""
    s = copy.copy(Q.methane_minimal())
    s.prim_exp, s.prim_coef, s.prim_pow = s.prim_exp[:-1].copy(), s.prim_coef[:-1].copy(), s.prim_pow[:-1].copy()
    s.ao_prim_off = s.ao_prim_off.copy()
    s.ao_prim_off[-1] -= 1
    return s


SPECS = {"four": Q.methane_minimal, "one": lambda: Q.methane_minimal(n_rot=1), "table": _table_driven}
W = 24577


@pytest.mark.parametrize("name", sorted(SPECS))
def test_large_batch_rows(ctx, oracle, name):
    spec = SPECS[name]()
    p = spec.params()
    p[8:] = 0.1 * np.arange(1, len(p) - 7)
    spec = spec.with_params(p)
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, W, seed=16)
    big = sysh.logderiv_batch(pos, el_derivs=True)
    only = sysh.logderiv_batch(pos)
    assert all(np.array_equal(a, b) for a, b in zip(big, only))
    for rows in (slice(0, 900), slice(W - 900, W)):
        small = sysh.logderiv_batch(pos[rows], el_derivs=True)
        dO, dE, dD = (np.linalg.norm(np.asarray(a)[rows] - b) for a, b in zip(big, small))
        size = np.linalg.norm(small[2])
        assert dO <= 1e-13 * np.linalg.norm(small[0])
        assert dE <= 1e-13 * size and dD <= 1e-13 * size, (dE, dD, size)
    O = oracle.log_derivatives(spec, pos[:200])
    assert np.linalg.norm(big[0][:200] - O) <= 1e-9 * np.linalg.norm(O)
    sysh.close()

"""SR rows of the compile-time CH4 layout and of MethaneGTO without rotations: a batch
above 9216 configurations goes a thread per walker, smaller ones by teams.  O_p against
the oracle (1e-9 of the norm), and E_L and dE_L/dp of the same configurations in a small
batch.  Both routes fill the orbital matrix in AO order with the same exponential and
divide by pivots, so configurations next to a node, which amplify that rounding, agree:
only sums of 64-bit terms differ, 1e-14 of the norm (95 pairs and 10 electrons of some
1e-16 each).  Next to a node E_L is what is left of electrons' terms as large as
dE_L/dp, so its difference is measured against those."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [Q.methane_gto, lambda: Q.methane_minimal(n_rot=0)], ids=["ch4_gto", "ch4_min"])
def test_rows_keep_their_rounding(ctx, oracle, make):
    spec = make()
    sysh = Q.System(ctx, spec)
    pos = random_configs(spec, 9217, seed=6)
    big = sysh.logderiv_batch(pos, el_derivs=True)
    for r0 in (0, 4000, 9217 - 1500):
        rows = slice(r0, r0 + 1500)
        small = sysh.logderiv_batch(pos[rows], el_derivs=True)
        dO, dE, dD = (np.linalg.norm(np.asarray(a)[rows] - b) for a, b in zip(big, small))
        size = np.linalg.norm(small[2])
        assert dO <= 1e-14 * np.linalg.norm(small[0])
        assert dE <= 1e-14 * size and dD <= 1e-14 * size, (dE, dD, size)
    O = oracle.log_derivatives(spec, pos[:200])
    assert np.linalg.norm(np.asarray(big[0])[:200] - O) <= 1e-9 * np.linalg.norm(O)
    sysh.close()

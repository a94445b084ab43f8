"""The Jastrow part of d ln|psi|/dR to 64 bits: with amplitudes A of 1000 it carries the
force, and what A = 0 gives is the determinant's part.  Against numpy's divisions: a
term takes some six roundings (1e-15 together), the sum over ten electrons a few more:
2e-15 of the norm, where reciprocals of 1e-14 leave more."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [Q.methane_gto, Q.methane_minimal])
def test_jastrow_force(ctx, make):
    spec = make()
    pos = random_configs(spec, 64, seed=5)
    om = []
    for A in (1000.0, 0.0):
        p = spec.params()
        p[6:8] = A
        s = Q.System(ctx, spec.with_params(p))
        om.append(s.forces_batch(pos)[1])
        s.close()
    want = np.zeros_like(om[0])
    for I in range(spec.n_nuc):
        d = (pos - spec.nuc_pos[I]).astype(np.longdouble)
        r = np.sqrt((d * d).sum(2, keepdims=True))
        f = 1000.0 * spec.nuc_charge[I] / (r * (1 + spec.jas[4 + spec.nuc_species[I]] * r) ** 2)
        want[:, I] = (f * d).sum(1)
    err = np.linalg.norm(om[0] - om[1] - want) / np.linalg.norm(want)
    assert err <= 2e-15, err

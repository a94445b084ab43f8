"""FP64 evaluation of the electron gas: the Jastrow sum over 1431 pairs has the rounding
of 64 bits and no drift.  A configuration's log|psi| and the oracle's each carry some
1e-13 of rounding, which goes either way; over 200 configurations their mean difference
stays below 2e-13, where reciprocals of 1e-14 that err to one side give 1.3e-12."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["rpa", "pade", "yukawa"])
def test_log_psi_has_no_drift(ctx, oracle, form):
    spec = Q.electron_gas(form=form)
    sysh = Q.System(ctx, spec)
    pos = np.random.default_rng(7).uniform(0.0, spec.box_L, size=(200, 54, 3))
    d = sysh.eval_batch(pos)["logabs"] - oracle.evaluate(spec, pos)["logabs"]
    assert abs(d.mean()) <= 2e-13, d.mean()
    assert np.median(np.abs(d)) <= 1e-12
    sysh.close()

"""Electron gas at positions outside the box (set_positions does not wrap them): E_L
and log|psi| of a refresh at the walkers' own positions against the oracle, 1e-6 as
for every refresh of FP32 walkers (their coordinates carry FP32's rounding, which the
comparison takes over); FP64 walkers 1e-8 and 1e-9 (the outer images are summed in FP32
for both)."""
import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [L.QMC_FP32_REFINE, L.QMC_FP64])
@pytest.mark.parametrize("boxes", [1, 3, 20])
def test_refresh_of_unwrapped_positions(ctx, oracle, boxes, prec):
    spec = Q.electron_gas()
    rng = np.random.default_rng(boxes)
    W = 24
    pos = spec.box_L * (rng.random((W, 54, 3)) + rng.integers(-boxes, boxes + 1, (W, 54, 3)))
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, prec)
    wk.set_positions(pos)
    wk.refresh()
    want = oracle.evaluate(spec, wk.get_positions())
    la, _, el = wk.state()
    assert np.max(np.abs(el - want["e_local"])) <= (1e-6 if prec == L.QMC_FP32_REFINE else 1e-8)
    assert np.max(np.abs(la - want["logabs"])) <= (1e-6 if prec == L.QMC_FP32_REFINE else 1e-9)
    wk.close()
    sysh.close()

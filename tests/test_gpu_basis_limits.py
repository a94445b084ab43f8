"""A basis beyond a shape's tables is refused by every call, in either precision and at
any size: Li whose two orbitals do not share their seven exponents (14 primitives in
shells of their own, the shape has 8)."""
import copy

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.helpers import random_configs

pytestmark = pytest.mark.gpu


def test_too_many_primitives(ctx):
    spec = copy.copy(Q.lithium_atom())
    spec.prim_exp = spec.prim_exp * np.r_[np.ones(7), np.full(7, 1.1)]
    sysh = Q.System(ctx, spec)
    for W in (3, 9217):
        pos = random_configs(spec, W, seed=1)
        for call in (lambda: sysh.eval_batch(pos), lambda: sysh.forces_batch(pos)):
            with pytest.raises(L.QMCError):
                call()
        for prec in (L.QMC_FP64, L.QMC_FP32_REFINE):
            wk = Q.Walkers(sysh, W, prec)
            wk.set_positions(pos)
            for call in (wk.refresh, lambda: wk.sweep(L.QMC_MOVE_ONE_GAUSS, 1, 0, seed=1, step=0.1),
                         lambda: wk.sweep(L.QMC_MOVE_ALL_GAUSS, 1, 0, seed=1, step=0.1)):
                with pytest.raises(L.QMCError):
                    call()
            wk.close()
    sysh.close()

"""Electron-gas refreshes of two threads, each with a context and a reciprocal cutoff of
its own (the refresh's shared memory grows with the cutoff)."""
import threading

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def test_two_cutoffs_at_once(oracle):
    out, start = {}, threading.Barrier(2)

    def work(kmax):
        try:
            ctx = Q.Context(0)
            spec = Q.electron_gas(kmax=kmax)
            sysh = Q.System(ctx, spec)
            start.wait()
            for prec in (L.QMC_FP32_REFINE, L.QMC_FP64):
                wk = Q.Walkers(sysh, 4, prec)
                wk.init(seed=kmax)
                wk.refresh()
                batch = Q.Batch(ctx, [wk])
                batch.refresh()
                out[kmax, prec] = wk.get_positions(), wk.state()[2]
                batch.close()
                wk.close()
            sysh.close()
            ctx.close()
        except Exception as e:                                       # noqa: BLE001
            out["error", kmax] = e

    threads = [threading.Thread(target=work, args=(k,)) for k in (2, 9)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not [v for k, v in out.items() if k[0] == "error"], out
    for (kmax, _), (pos, el) in out.items():
        assert np.max(np.abs(el - oracle.evaluate(Q.electron_gas(kmax=kmax), pos)["e_local"])) <= 1e-6


def test_largest_cutoff(ctx):
    """|n| <= 9 has 1535 half-space vectors; 10 has 2084, more than the table holds."""
    for kmax, ok in ((9, True), (10, False)):
        sysh = Q.System(ctx, Q.electron_gas(kmax=kmax))
        wk = Q.Walkers(sysh, 2, L.QMC_FP64)
        if ok:
            wk.init(seed=1)
            wk.refresh()
        else:
            with pytest.raises(L.QMCError):
                wk.init(seed=1)
        wk.close()
        sysh.close()

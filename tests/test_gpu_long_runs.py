"""vmc_run with all-electron moves over more steps than its partial sums hold at once
(256 MiB of 16 bytes a block and step): the device memory it takes is bounded, a shorter
run is a prefix of a longer one, and the steps around the edge are the single steps'."""
import ctypes as C
import threading

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.test_zz_no_alloc import _cudart

pytestmark = pytest.mark.gpu

W, KW = 4864, dict(n_walkers=4864, move_kind=L.QMC_MOVE_ALL_BOX, step=1.0, seed=3)
ROWS = (256 << 20) // (16 * (W // 8))          # eight H2 walkers a block: 27 594 steps


def test_steps_across_the_edge(ctx):
    sysh = Q.System(ctx, Q.h2_mo())
    long = Q.vmc_run(sysh, n_steps=ROWS + 40, **KW)["energies"]
    short = Q.vmc_run(sysh, n_steps=60, **KW)["energies"]
    assert len(long) == ROWS + 40 and np.array_equal(long[:60], short)
    wk = Q.Walkers(sysh, W, L.QMC_FP64)
    wk.init(seed=3)
    wk.refresh()
    wk.sweep(L.QMC_MOVE_ALL_BOX, ROWS - 3, 0, seed=3, step=1.0)
    for t in range(ROWS - 3, ROWS + 5):
        wk.sweep(L.QMC_MOVE_ALL_BOX, 1, t, seed=3, step=1.0)
        # the same decisions but for one within rounding of its threshold: some 1e8 were taken
        assert abs(long[t] - wk.state()[2].mean()) <= 1e-2
    wk.close()
    sysh.close()


def test_device_memory_of_a_long_run_is_bounded(ctx):
    rt = _cudart()
    sysh = Q.System(ctx, Q.h2_mo())

    def free_bytes():
        f, t = C.c_size_t(), C.c_size_t()
        assert rt.cudaMemGetInfo(C.byref(f), C.byref(t)) == 0
        return f.value

    Q.vmc_run(sysh, n_steps=10, **KW)
    start, low, done = free_bytes(), [1 << 62], threading.Event()

    def watch():
        while not done.is_set():
            low[0] = min(low[0], free_bytes())

    th = threading.Thread(target=watch)
    th.start()
    r = Q.vmc_run(sysh, n_steps=200000, **KW)
    done.set()
    th.join()
    assert len(r["energies"]) == 200000
    assert start - low[0] <= 600 << 20, start - low[0]
    sysh.close()

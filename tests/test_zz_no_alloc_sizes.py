"""qmc_sr_sums_noalloc up to the sizes that qmc.h states,
2 (2 + 2P + P(P+1)/2) ceil(W/256) <= 65536, and one walker beyond them.
Compensated 64-bit sums: 1e-14 of the sum of magnitudes."""
import ctypes as C

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L
from tests.test_zz_no_alloc import DevBuf, _cudart

pytestmark = pytest.mark.gpu


def _call(lib, W, P, dE, dO, dS):
    p = lambda b: C.cast(b.ptr, C.POINTER(C.c_double))
    return lib.qmc_sr_sums_noalloc(p(dE), p(dO), W, P, p(dS), None)


@pytest.mark.parametrize("W, P", [(5000, 12), (20000, 12), (80640, 12), (49152, 16), (300000, 1)])
def test_documented_sizes(ctx, W, P):
    lib, rt = Q.load_library(), _cudart()
    rng = np.random.default_rng(W + P)
    E, O = rng.standard_normal(W) - 3.0, rng.standard_normal((W, P))
    M = 2 + 2 * P + P * (P + 1) // 2
    bufs = dE, dO, dS = DevBuf(rt, 8 * W), DevBuf(rt, 8 * W * P), DevBuf(rt, 8 * M)
    try:
        dE.put(E)
        dO.put(O)
        assert _call(lib, W, P, dE, dO, dS) == L.QMC_OK
        assert rt.cudaDeviceSynchronize() == 0
        cols = [E, E * E] + [O[:, p] for p in range(P)] + [E * O[:, p] for p in range(P)]
        cols += [O[:, p] * O[:, q] for p in range(P) for q in range(p, P)]
        want = np.array([c.astype(np.longdouble).sum() for c in cols], dtype=float)
        size = np.array([np.abs(c).sum() for c in cols])
        assert np.all(np.abs(dS.get(M) - want) <= 1e-14 * size)
    finally:
        for b in bufs:
            b.free()


def test_one_walker_more_is_refused(ctx):
    lib, rt = Q.load_library(), _cudart()
    b = DevBuf(rt, 8 * 80641 * 12)
    try:
        assert _call(lib, 80641, 12, b, b, b) == L.QMC_ERR_ARG
    finally:
        b.free()

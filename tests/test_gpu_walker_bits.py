"""FP32 walkers keep their bits: a chain's decisions follow from every rounding of the
sweeps and of the refreshed inverses, so kernels that lay out or pack the same operations
differently have to leave the same walkers.

The recorded values are the CRC-32 of the positions (FP32 words) and the accepted moves
after Gaussian sweeps, a refresh and further sweeps, as the kernels with one value per
instruction and shells from tables left them; starting points are multiples of 2^-10 about
the nuclei (in the box), so that no random generator enters.  A change that is meant to
round differently has to replace them.

Li and 6-31G CH4 sets by themselves run sweeps with their shells unrolled, in a batch the
table-driven ones: the same walkers, compared directly."""
import zlib

import numpy as np
import pytest

import rust_qmc_gb300 as Q
from rust_qmc_gb300 import _lib as L

pytestmark = pytest.mark.gpu

SPECS = {"c6h6": Q.benzene_minimal, "c6h6_gto": Q.benzene_gto, "heg_rpa": Q.electron_gas,
         "heg_pade": lambda: Q.electron_gas(form="pade"), "heg_twist": lambda: Q.electron_gas(twist=(0.25, 0.1, 0.4)),
         "ch4_min": Q.methane_minimal, "ch4_gto": Q.methane_gto, "li": Q.lithium_atom}
RECORDED = {
    "c6h6": [(30835, 1416568129), (29987, 1671903026), (49874, 3629297403)],
    "c6h6_gto": [(32898, 3012762340), (32506, 945654862), (49901, 2435163335)],
    "ch4_gto": [(8583, 504502631), (8358, 3103863477), (11914, 821556419)],
    "ch4_min": [(7927, 4226992770), (7750, 3526820182), (11931, 1699012003)],
    "heg_pade": [(21440, 999280827), (12657, 534244127), (44252, 587460150)],
    "heg_rpa": [(22235, 951712232), (14138, 1838774653), (45892, 3244888161)],
    "heg_twist": [(22559, 1353017995), (14751, 80737285), (45901, 247386820)],
    "li": [(2601, 4021587630), (2707, 55211686), (3603, 3661308190)],
}


def start(spec, W):
    k = np.arange(W * spec.n_elec * 3, dtype=np.uint64)
    u = ((k * np.uint64(2654435761) + (k * k * k) * np.uint64(40503)) >> np.uint64(7)) % np.uint64(1024)
    u = (u.astype(np.float64) / 1024.0).reshape(W, spec.n_elec, 3)
    if spec.box_L > 0:
        return np.float32(spec.box_L * u).astype(np.float64)
    centre = np.array([spec.nuc_pos[i] if i >= 0 else np.zeros(3) for i in spec.init_nuc])
    return np.float32(centre[None] + 2.0 * u - 1.0).astype(np.float64)


def chain(ctx, name, W):
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    wk = Q.Walkers(sysh, W, L.QMC_FP32_REFINE)
    wk.set_positions(start(spec, W))
    wk.refresh()
    step = 2.0 if spec.box_L > 0 else 0.3
    out = []
    for t, move in ((0, L.QMC_MOVE_ONE_GAUSS), (4, L.QMC_MOVE_ONE_GAUSS), (8, L.QMC_MOVE_ONE_DRIFT)):
        acc = wk.sweep(move, 4, t, seed=77, step=step, tau=0.005, max_drift=1.0)
        out.append((acc, zlib.crc32(np.float32(wk.get_positions()).tobytes())))
        wk.refresh()
    wk.close()
    sysh.close()
    return out


@pytest.mark.parametrize("name", sorted(SPECS))
def test_chain_bits(ctx, name):
    assert chain(ctx, name, 301) == RECORDED[name]


@pytest.mark.parametrize("name", ["li", "ch4_gto", "ch4_min"])
@pytest.mark.parametrize("W", [1, 130, 4097])
def test_batched_walkers_are_the_same(ctx, name, W):
    spec = SPECS[name]()
    sysh = Q.System(ctx, spec)
    a, b = (Q.Walkers(sysh, W, L.QMC_FP32_REFINE) for _ in range(2))
    for wk in (a, b):
        wk.set_positions(start(spec, W))
        wk.refresh()
    batch = Q.Batch(ctx, [a])
    for t in range(2):
        batch.run_steps(L.QMC_MOVE_ONE_GAUSS, 1, 5, 5 * t, 31, step=0.3)
        b.sweep(L.QMC_MOVE_ONE_GAUSS, 5, 5 * t, seed=Q.batch_system_seed(31, 0), step=0.3)
        b.refresh()
        assert np.array_equal(a.get_positions(), b.get_positions())
        assert all(np.array_equal(x, y) for x, y in zip(a.state(), b.state()))
    batch.close()
    a.close()
    b.close()
    sysh.close()

// qmc_shape_ch4min_measure.cu -- initialisation and measurement kernels for the ShapeCH4Min system shape.
#include "qmc_walker_kernels.cuh"

namespace qmc {
QMC_DEFINE_SHAPE_MEASURE(ch4min, ShapeCH4Min)

int shape_step_all_ch4(const HostSys& hs, DevWalkers& dw, int mk, int n, uint64_t s0, double step, uint64_t seed,
                       cudaStream_t st, double* partial);
// All-electron steps: this layout has team kernels of its own and shares the
// table-driven shape's thread-per-walker ones.
int shape_step_all_ch4min(const HostSys& hs, DevWalkers& dw, int mk, int n, uint64_t s0, double step, uint64_t seed,
                          cudaStream_t st, double* partial) {
    using Teams = ShapeOps<ShapeCH4Min>::Teams;
    if (dw.prec == 0 && (!partial || team_measures(dw.W)))
        return mk == MOVE_ALL_BOX ? Teams::steps<MOVE_ALL_BOX>(hs, dw, n, s0, step, seed, partial, st)
                                  : Teams::steps<MOVE_ALL_GAUSS>(hs, dw, n, s0, step, seed, partial, st);
    return shape_step_all_ch4(hs, dw, mk, n, s0, step, seed, st, partial);
}
int shape_step_blocks_ch4min(const DevWalkers& dw) { return ShapeOps<ShapeCH4Min>::step_blocks(dw); }
}  // namespace qmc

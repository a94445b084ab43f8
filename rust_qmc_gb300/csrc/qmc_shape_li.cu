// qmc_shape_li.cu -- all kernels for the ShapeLi system shape.
#include "qmc_walker_kernels.cuh"

namespace qmc {
QMC_DEFINE_SHAPE_MEASURE(li, ShapeLi)
QMC_DEFINE_SHAPE_ONE(li, ShapeLi)
QMC_DEFINE_SHAPE_ALL(li, ShapeLi)
QMC_DEFINE_SHAPE_BATCH_SWEEP(li, ShapeLi)
QMC_DEFINE_SHAPE_BATCH_MEASURE(li, ShapeLi)
int shape_sweep_gauss_li_sto7(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, uint64_t seed,
                              cudaStream_t st) {
    return ShapeOps<ShapeLiSto7>::template sweep_one<float, MOVE_ONE_GAUSS>(hs, dw, n, s0, step, 0.0, 0.0, seed, st);
}
}  // namespace qmc

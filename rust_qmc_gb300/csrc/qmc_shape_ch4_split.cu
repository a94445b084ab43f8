// qmc_shape_ch4_split.cu -- FP32 Gaussian sweeps of the ShapeCH4Split system shape.
#include "qmc_walker_kernels.cuh"

namespace qmc {
int shape_sweep_gauss_ch4_split(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, uint64_t seed,
                                cudaStream_t st) {
    return ShapeOps<ShapeCH4Split>::template sweep_one<float, MOVE_ONE_GAUSS>(hs, dw, n, s0, step, 0.0, 0.0, seed, st);
}
}  // namespace qmc

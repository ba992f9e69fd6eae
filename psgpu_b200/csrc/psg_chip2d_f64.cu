// psg_chip2d_f64.cu -- the on-chip 2D integrator's FP64 kernels (psg_chip2d_run.cuh)
#define PSG_CHIP2D_INSTANTIATE
#include "psg_chip2d_run.cuh"

namespace psg {
PSG_CHIP2D_TEMPLATES(double)
}  // namespace psg

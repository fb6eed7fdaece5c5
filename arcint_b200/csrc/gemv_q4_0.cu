// gemv_q4_0.cu -- the decode GEMV of Q4_0 weights (instantiation only, see gemv_launch.cuh).
#include "gemv_launch.cuh"

namespace b200q {

B200Q_GEMV_TYPE(, B200Q_TYPE_Q4_0)
B200Q_GEMV_TYPE_ONE(, B200Q_TYPE_Q4_0)
B200Q_GEMV_TYPE_AR(, B200Q_TYPE_Q4_0)
B200Q_GEMV_TYPE_FUSED(, B200Q_TYPE_Q4_0)

}  // namespace b200q

// gemv_q4_k.cu -- the decode GEMV of Q4_K weights (instantiation only, see gemv_launch.cuh).
#include "gemv_launch.cuh"

namespace b200q {

B200Q_GEMV_TYPE(, B200Q_TYPE_Q4_K)
B200Q_GEMV_TYPE_ONE(, B200Q_TYPE_Q4_K)
B200Q_GEMV_TYPE_AR(, B200Q_TYPE_Q4_K)

}  // namespace b200q

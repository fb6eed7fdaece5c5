// gemv_q5_k.cu -- the decode GEMV of Q5_K weights (instantiation only, see gemv_launch.cuh).
#include "gemv_launch.cuh"

namespace b200q {

B200Q_GEMV_TYPE(, B200Q_TYPE_Q5_K)
B200Q_GEMV_TYPE_ONE(, B200Q_TYPE_Q5_K)

}  // namespace b200q

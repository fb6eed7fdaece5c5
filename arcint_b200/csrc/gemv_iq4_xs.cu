// gemv_iq4_xs.cu -- the decode GEMV of IQ4_XS weights (instantiation only, see gemv_launch.cuh).
#include "gemv_launch.cuh"

namespace b200q {

B200Q_GEMV_TYPE(, B200Q_TYPE_IQ4_XS)
B200Q_GEMV_TYPE_AR(, B200Q_TYPE_IQ4_XS)

}  // namespace b200q

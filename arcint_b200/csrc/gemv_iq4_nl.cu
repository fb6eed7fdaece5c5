// gemv_iq4_nl.cu -- the decode GEMV of IQ4_NL weights (instantiation only, see gemv_launch.cuh).
#include "gemv_launch.cuh"

namespace b200q {

B200Q_GEMV_TYPE(, B200Q_TYPE_IQ4_NL)

}  // namespace b200q

// Integer tensor-core matvec, 4-bit weight codes.
#include "common.cuh"

namespace b200q {
B200Q_DEFINE_STATUS_WORD(gemv_i8_q4_read_status)
}

#include "gemv_i8.cuh"

namespace b200q {
int gemv_i8_q4(const GemvParams& p, bool gate_up, cudaStream_t stream) { return dispatch_i8<4>(p, gate_up, stream); }
}

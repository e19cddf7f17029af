// Label smooth, rows of up to 2048 channels: backward and the fused training step (rows_short.cuh).
#include "rows_short.cuh"

namespace b200 {
int launch_rows_lsr_bwd(int dtype, const SoftmaxParams &prm, cudaStream_t stream) {
    return launch_rows_dtype<kLSR, true>(dtype, prm, stream);
}
}  // namespace b200

// Large margin, rows of up to 2048 channels: backward and the fused training step (rows_short.cuh).
#include "rows_short.cuh"

namespace b200 {
int launch_rows_lmargin_bwd(int dtype, const SoftmaxParams &prm, cudaStream_t stream) {
    return launch_rows_dtype<kLMargin, true>(dtype, prm, stream);
}
}  // namespace b200

// Large margin, rows of up to 2048 channels: forward (rows_short.cuh).
#include "rows_short.cuh"

namespace b200 {
int launch_rows_lmargin_fwd(int dtype, const SoftmaxParams &prm, cudaStream_t stream) {
    return launch_rows_dtype<kLMargin, false>(dtype, prm, stream);
}
}  // namespace b200

// What the launchers of the softmax-family kernels hand to each other.
#pragma once

#include "softmax_core.cuh"

namespace b200 {

struct SoftmaxParams {
    const void *logits;
    const int64_t *labels;
    void *losses;            // [N, M] dtype or null
    void *grads;             // [N, C, M] dtype (backward)
    const void *grad_out;    // see grad_mode
    int grad_mode;
    const double *denom;
    void *workspace;
    ReduceRecord *out;
    float4 *stats;           // [N*M] per-pixel statistics: written by the chunked forward, read by
                             // the chunked backward (null: not wanted / not available)
    int64_t N, C, M;
    int64_t ignore;
    LossConsts k;
    // tile geometry
    int TP, KS, CB, nbox, rows;
    int nbx;                 // boxes of TP pixels per tile (pair kernel)
    int stages;              // ring depth of the pipelined kernels
    int64_t tiles_per_image, total_tiles;
    int defer;               // cross-GPU sum of the fused step: post only (see grid_reduce_finish)
    int after_count;         // fused step launched as a programmatic dependent of the label count
    const float *chan_w;     // kPC: class weights [C] (device)
};

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// M == 1 layouts whose rows are kept in registers (rows_short.cuh; one translation unit per loss and
// direction): forward (bwd = false; prm.losses and / or prm.out), backward (prm.out null) and the
// fused training step (prm.out given).
constexpr int kShortRowsMaxC = 2048;
// rows of whole 16-byte vectors from here on go warp by row (rows_vec_kernel): 128 channels
// float32 / bfloat16 step 36.5 / 40.0 us there against 30.3 / 32.8 us in rows_short_kernel
// ([131072, 128]), 256 channels 25.5 / 22.6 against 32.0 / 33.6 us ([65536, 256])
constexpr int kVecMinC = 256;
bool short_rows_eligible(size_t es, const void *logits, const void *io, const void *labels, int64_t N, int64_t C,
                         int64_t M);
int launch_short_rows(int kind, bool bwd, int dtype, const SoftmaxParams &prm, cudaStream_t stream);

}  // namespace b200

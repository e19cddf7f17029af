// M == 1 with up to 2048 channels: [N, C] classification inputs and channels-last images, where every
// pixel is a row of C contiguous logits.  A row crosses HBM once and is held in REGISTERS from its
// load to its gradient; two kernels, by what a row's length and alignment allow:
//
//   rows_vec_kernel    rows of 256 or more channels in whole 16-byte vectors: a warp owns a row, streams it from
//                      global memory into registers and its gradient back, the next row's
//                      vectors in flight under the arithmetic.  No shared memory.
//   rows_short_kernel  every other row (any C, any element alignment): a stage is a contiguous run of
//                      rows moved by one bulk copy in and (backward) one out; TPR adjacent lanes
//                      share a row, read it from the stage ONCE as packed pairs and leave the
//                      gradient there once.
//
// Both were bound by instruction issue when a row stayed in shared memory and was walked three times
// (35 thread instructions per bfloat16 element).  Measured, before -> after, kernel time:
//   bfloat16 [32768, 1000] label-smooth step                  69.9 -> 30 us (4.4 TB/s)
//   half [894916, 150] large margin, forward / backward       176 / 334 -> 95 / 160 us
//
// `prm.out` given: loss sum and count are reduced over the grid (the forward's record, or in backward
// the fused training step).  Included by one translation unit per loss and direction.
#pragma once

#include <type_traits>

#include "pipeline.cuh"
#include "softmax_params.cuh"

namespace b200 {
namespace {

constexpr int kShortCompute = 256;
constexpr int kShortBlock = kShortCompute + 64;
constexpr int kShortPairs = 20;
constexpr int kVecThreads = 256;
constexpr int kVecWarps = kVecThreads / 32;

// ---- one row's mathematics on packed pairs (softmax_core.cuh has the formulas).  `each(f)` calls
// f(pair) for every pair this lane holds, `tail` (singles only) adds the odd element.

// Largest value over the lanes of a row.
__device__ __forceinline__ float lanes_max(float m, int tpr, unsigned mask) {
    for (int o = tpr >> 1; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(mask, m, o));
    return m;
}
__device__ __forceinline__ float lanes_sum(float s, int tpr, unsigned mask) {
    for (int o = tpr >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o);
    return s;
}

// Large margin after the sums: the row's loss and the coefficients of its gradient
// g_j = q_j (A + B d_j) + Cc with q_j = e^{d_j} / s', and of the target, -r.  `lbi` < 0: a label outside
// the classes (undefined in the reference): every channel counts as off target.  `xd`: the value that
// stood in for the target in the sums; its terms come back out here (s' >= 1 >= e^{xd - m'}, so nothing cancels).
// `sd`: the sum of the differences d_j = x_j - m' -- of the logits themselves it would carry an offset that they share.
// The stand-in is the larger of two channels: a channel masked with the type's lowest value, added twice, would
// overflow the sum.
struct MarginRow {
    float loss, inv_s, sqx, r;
    __device__ __forceinline__ void finish(float m, float s, float sde, float sd, float xl, float xd, int lbi,
                                           const LossConsts &k) {
        if (lbi >= 0) {
            const float dc = xd - m, ec = ex2f(dc * kLog2e);
            s -= ec;
            sde -= dc * ec;
            sd -= dc;
        }
        inv_s = __fdividef(1.f, s);
        sqx = sde * inv_s;
        const float mm = fmaxf(m, xl);
        const float e_no = s * ex2f((m - mm) * kLog2e);
        const float e_lb = ex2f((xl - mm) * kLog2e);
        const float s_all = e_no + e_lb;
        r = __fdividef(e_no, s_all);
        loss = (mm + __logf(s_all)) - xl + k.half_lam * (sqx - k.a * sd);
    }
};

// The factor c of x c - m c in the exponent of 2: log2 e, or where m c would overflow one half -- logits that far
// out are equal or 2^100 apart, so e^{x - m} is 1 or 0 either way.  (Rows of an odd length only, where such logits
// have always been taken; the two registers cost 16-bit rows of even length 2 %.)
__device__ __forceinline__ float exponent_scale(float m) { return fabsf(m) < 2.3e38f ? kLog2e : 0.5f; }

// Two adjacent 16-bit elements in a word.
template <typename T> struct Two;
template <> struct Two<__half> { using type = __half2; };
template <> struct Two<__nv_bfloat16> { using type = __nv_bfloat162; };
template <typename T> __device__ __forceinline__ uint32_t max_words(uint32_t a, uint32_t b) {
    using V = typename Two<T>::type;
    const V m = __hmax2(*reinterpret_cast<V *>(&a), *reinterpret_cast<V *>(&b));
    return *reinterpret_cast<const uint32_t *>(&m);
}
template <typename T> __device__ __forceinline__ pk_t word_pk(uint32_t w) { return ld_pk(reinterpret_cast<const T *>(&w)); }

// Shared-memory accesses by 32-bit address.
__device__ __forceinline__ uint32_t lds_word(uint32_t a) {
    uint32_t w;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(a) : "memory");
    return w;
}
__device__ __forceinline__ uint32_t lds_two(uint32_t a, uint32_t b) {     // two 16-bit elements into a word
    unsigned short x, y;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(a) : "memory");
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(y) : "r"(b) : "memory");
    return uint32_t(x) | uint32_t(y) << 16;
}
template <typename T> __device__ __forceinline__ pk_t lds_pk(uint32_t a) {
    if constexpr (sizeof(T) == 4) {
        pk_t r;
        asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r) : "r"(a) : "memory");
        return r;
    } else {
        unsigned w;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(a) : "memory");
        return ld_pk(reinterpret_cast<const T *>(&w));
    }
}
template <typename T> __device__ __forceinline__ void sts_pk(uint32_t a, pk_t v) {
    if constexpr (sizeof(T) == 4) {
        asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
    } else {
        unsigned w;
        st_pk(reinterpret_cast<T *>(&w), v);
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(w) : "memory");
    }
}
template <typename T> __device__ __forceinline__ float lds_one(uint32_t a) {
    if constexpr (sizeof(T) == 4) {
        float r;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(a) : "memory");
        return r;
    } else {
        unsigned short h;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(a) : "memory");
        return to_f32(*reinterpret_cast<const T *>(&h));
    }
}
template <typename T> __device__ __forceinline__ void sts_one(uint32_t a, float v) {
    if constexpr (sizeof(T) == 4) {
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
    } else {
        const T x = from_f32<T>(v);
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(*reinterpret_cast<const unsigned short *>(&x)) : "memory");
    }
}

// ------------------------------------------------------------------------------------ rows_short
// NP: pairs a lane can hold.  MODE: what a lane's unit is and how it walks its units (t, t + TPR, ...).
//   kSingles  odd C: a unit is one element, a pair is two of the lane's units
//   kPairs    even C: a unit is an adjacent pair, one 4- or 8-byte access
//   kRotated  the same where C is a multiple of 4 and few lanes share a row: the rows of a warp lie an
//             even number of words apart and would share banks, so each row's walk starts at a unit
//             that depends on the row and wraps around
enum RowWalk { kSingles = 0, kPairs = 1, kRotated = 2 };

// 16-bit types hold the row as the words they were read as (half the registers, so three blocks on an SM
// instead of two) and convert in each sweep, unless the gradient wants the exponentials themselves.
template <typename T, int KIND, bool BWD> constexpr bool hold_words() {
    return sizeof(T) == 2 && (KIND == kLMargin || !BWD);
}
template <typename T, int KIND, bool BWD, int NP> constexpr int short_blocks() {   // blocks per SM (registers)
    if (NP <= 4) return 4;
    if (NP <= 12) return 3;
    if (NP <= 20) return sizeof(T) == 2 ? 3 : 2;
    return hold_words<T, KIND, BWD>() ? 2 : 1;
}
template <typename T, int KIND, bool BWD, int MODE, int NP>
__global__ void __launch_bounds__(kShortBlock, short_blocks<T, KIND, BWD, NP>())
rows_short_kernel(const SoftmaxParams prm) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ PipeBarriers bars;
    __shared__ double sh_red[64];

    // every lane holds at least NU of the NP pairs (launch_rows_short picks the smallest NP of 4, 8, 10,
    // 12, 16, 20, 32 that holds a row): no check on those, so that their loads go out back to back
    constexpr int NU = NP <= 4 ? 0 : NP <= 20 ? NP - 4 : 20;
    constexpr bool PAIRED = MODE != kSingles, kHold = hold_words<T, KIND, BWD>();
    const int C = static_cast<int>(prm.C), NS = prm.stages, TPR = prm.KS;
    const int R = kShortCompute / TPR, G = prm.rows;         // rows per group, groups per stage
    const int RS = R * G;
    unsigned char *base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const size_t label_off = (size_t(RS) * C * sizeof(T) + 127) & ~size_t(127);
    const size_t stage_bytes = label_off + size_t(RS) * sizeof(int64_t);
    const int tid = threadIdx.x;
    const bool reduce = prm.out != nullptr;
    unsigned *status = prm.workspace ? reinterpret_cast<unsigned *>(prm.workspace) + 1 : nullptr;
    const int n_stages = int((prm.N + RS - 1) / RS);         // (RS >= 8 rows: the count fits 32 bits)
    const uint32_t full_bytes = uint32_t(RS) * C * sizeof(T);

    pipe_init<kShortCompute, BWD>(bars, NS);
    const int first = blockIdx.x, stride = gridDim.x;
    double acc_loss = 0.0;
    int acc_cnt = 0;                                         // rows this thread counted

    if (tid == kShortCompute) {
        int k = 0;
        for (int st = first; st < n_stages; st += stride, ++k) {
            const int s = k % NS;
            if (k >= NS && !mbar_wait_bounded(&bars.empty[s], ((k / NS) - 1) & 1, status)) break;
            const int64_t row0 = int64_t(st) * RS;
            if (prm.N - row0 >= RS) {
                unsigned char *stage = base + s * stage_bytes;
                const unsigned char *src = static_cast<const unsigned char *>(prm.logits) + row0 * C * sizeof(T);
                mbar_expect_tx(&bars.full[s], full_bytes + uint32_t(RS) * sizeof(int64_t));
                for (uint32_t off = 0; off < full_bytes; off += 32768u) {
                    const uint32_t nb = full_bytes - off < 32768u ? full_bytes - off : 32768u;
                    bulk_load_1d(stage + off, src + off, nb, &bars.full[s]);
                }
                bulk_load_1d(stage + label_off, prm.labels + row0, uint32_t(RS) * sizeof(int64_t), &bars.full[s]);
            } else {
                mbar_expect_tx(&bars.full[s], 0);            // ragged end: the compute threads fetch it themselves
            }
        }
    } else if (BWD && tid == kShortCompute + 32) {
        int k = 0;
        for (int st = first; st < n_stages; st += stride, ++k) {
            const int s = k % NS;
            if (!mbar_wait_bounded(&bars.ready[s], (k / NS) & 1, status)) break;
            const int64_t row0 = int64_t(st) * RS;
            if (prm.N - row0 >= RS) {
                const unsigned char *stage = base + s * stage_bytes;
                unsigned char *dst = static_cast<unsigned char *>(prm.grads) + row0 * C * sizeof(T);
                for (uint32_t off = 0; off < full_bytes; off += 32768u) {
                    const uint32_t nb = full_bytes - off < 32768u ? full_bytes - off : 32768u;
                    bulk_store_1d(dst + off, stage + off, nb);
                }
                bulk_commit();
                bulk_wait_read_all();
            }
            mbar_arrive(&bars.empty[s]);
        }
        bulk_wait_all();
    } else if (tid < kShortCompute) {
        const int lane = tid & 31;
        const int t = tid & (TPR - 1);                       // my lane inside the row (TPR is a power of two)
        const int row_of = tid >> (31 - __clz(TPR));
        const unsigned row_mask = (TPR == 32 ? 0xffffffffu : ((1u << TPR) - 1u)) << (lane & ~(TPR - 1));
        const int units = PAIRED ? C >> 1 : C;
        const int cnt = (units - t + TPR - 1) >> (31 - __clz(TPR));
        const int np = PAIRED ? cnt : cnt >> 1;
        const bool odd = !PAIRED && (cnt & 1);
        const int step = (PAIRED ? 2 : 1) * TPR;             // elements between my units
        const T *gout = static_cast<const T *>(prm.grad_out);
        T *losses = static_cast<T *>(prm.losses);
        const LossConsts kc = prm.k;
        float gscale = 1.f;
        if (BWD && reduce) pdl_wait();                       // the divisor comes from the label count in front
        if (BWD) gscale = uniform_grad_scale(prm.grad_out, prm.grad_mode, prm.denom);
        int k = 0;
        for (int st = first; st < n_stages; st += stride, ++k) {
            const int s = k % NS;
            bool ok = true;
            if (lane == 0) ok = mbar_wait_bounded(&bars.full[s], (k / NS) & 1, status);
            // (the ragged last stage needs all compute threads at a named barrier, which has no
            // time limit: every stage's decision to go on is taken by all of them together)
            if (!compute_all(ok, kShortCompute)) break;
            const int64_t row0 = int64_t(st) * RS;
            const int nrows = prm.N - row0 >= RS ? RS : int(prm.N - row0);
            const bool ragged = nrows < RS;
            T *tile = reinterpret_cast<T *>(base + s * stage_bytes);
            int64_t *tile_labels = reinterpret_cast<int64_t *>(base + s * stage_bytes + label_off);
            if (ragged) {
                const T *src = static_cast<const T *>(prm.logits) + row0 * C;
                for (int e = tid; e < nrows * C; e += kShortCompute) tile[e] = src[e];
                for (int e = tid; e < nrows; e += kShortCompute) tile_labels[e] = prm.labels[row0 + e];
                compute_sync(kShortCompute);
            }
            for (int rowl = row_of; rowl < nrows; rowl += R) {
                const int64_t row = row0 + rowl;
                const int64_t lb = tile_labels[rowl];
                const bool valid = lb != prm.ignore;
                const int lbi = (lb >= 0 && lb < C) ? int(lb) : -1;
                T *rp = tile + size_t(rowl) * C;
                if (!valid) {
                    if (!BWD && losses && t == 0) losses[row] = from_f32<T>(0.f);
                    if (BWD)
                        for (int p = t; p < C; p += TPR) rp[p] = from_f32<T>(0.f);
                    continue;
                }
                T up{};
                if (BWD && prm.grad_mode == 2) up = gout[row];        // (used after the sums)
                const int lunit = PAIRED ? lbi >> 1 : lbi;
                const bool owner = lbi >= 0 && (lunit & (TPR - 1)) == t;      // my walk visits the label's unit
                float xl = 0.f, xd = 0.f;
                if (lbi >= 0) xl = to_f32(rp[lbi]);
                T dup{};
                if (KIND == kLMargin && lbi >= 0) {
                    // the target's place holds another channel's logit during the sums
                    const int c0 = (lbi == 0 && C > 1) ? 1 : 0, c1 = C > 2 ? (lbi <= 1 ? 2 : 1) : c0;
                    dup = rp[c0];
                    const T other = rp[c1];
                    if (to_f32(other) > to_f32(dup)) dup = other;
                    xd = to_f32(dup);
                }
                // every lane of the row has read x_lb before its owner writes there: the stand-in now or the
                // gradient later (shuffles in between do not order memory)
                if (KIND == kLMargin || BWD) __syncwarp(row_mask);
                if constexpr (KIND == kLMargin) {
                    if (lbi < 0) xl = kNegInf;
                    else if (owner) rp[lbi] = dup;
                }
                // a walk over my units: `w` is where it stands, `left` the units before a rotated one wraps
                const int rot = MODE == kRotated ? rowl % cnt : 0;
                const T *const w0 = rp + (PAIRED ? 2 : 1) * t + rot * step;
                struct Walk {
                    uint32_t w;
                    int left;
                };
                auto begin = [&] {
                    Walk k{smem_u32(w0), cnt - rot};
                    // (opaque: the gradient's walk makes its addresses anew instead of holding the first one's in registers)
                    asm volatile("" : "+r"(k.w));
                    return k;
                };
                auto next = [&](Walk &k) {
                    const uint32_t here = k.w;
                    k.w += uint32_t(step) * uint32_t(sizeof(T));
                    if (MODE == kRotated && --k.left == 0) k.w -= uint32_t(cnt) * uint32_t(step) * uint32_t(sizeof(T));
                    return here;
                };
                auto put = [&](Walk &walk, int i, pk_t g) {
                    if constexpr (PAIRED) {
                        const uint32_t at = next(walk);
                        if (i < NU || i < np) sts_pk<T>(at, g);
                    } else {
                        const float2 g2 = upk2(g);
                        const uint32_t at0 = next(walk), at1 = next(walk);
                        if (i < NU || i < np) {
                            sts_one<T>(at0, g2.x);
                            sts_one<T>(at1, g2.y);
                        }
                    }
                };
                T *const last = rp + t + (cnt - 1) * step;                // (singles: my odd element)
                pk_t v[NP];                                           // (the one of the two that is used)
                uint32_t held[NP];
                auto x_of = [&](int i) {
                    if constexpr (kHold) return word_pk<T>(held[i]);
                    else return v[i];
                };
                float vt = 0.f, m = kNegInf;
                if constexpr (kHold) {
                    Walk walk = begin();
                    constexpr uint32_t kLowest = std::is_same<T, __half>::value ? 0xfc00fc00u : 0xff80ff80u;   // -inf, twice
                    uint32_t w0 = kLowest, w1 = kLowest;
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        held[i] = kLowest;
                        if constexpr (PAIRED) {
                            const uint32_t at = next(walk);
                            if (i < NU || i < np) held[i] = lds_word(at);
                        } else {
                            const uint32_t at0 = next(walk), at1 = next(walk);
                            if (i < NU || i < np) held[i] = lds_two(at0, at1);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < NP; i += 2) {
                        w0 = max_words<T>(w0, held[i]);
                        w1 = max_words<T>(w1, held[i + 1]);
                    }
                    const float2 m2 = upk2(word_pk<T>(max_words<T>(w0, w1)));
                    m = fmaxf(m, fmaxf(m2.x, m2.y));
                    if (odd) {
                        vt = to_f32(*last);
                        m = fmaxf(m, vt);
                    }
                } else {
                    Walk walk = begin();
                    float2 m2 = splat2(kNegInf), m3 = m2;        // (two chains each: latency)
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        v[i] = psplat(-INFINITY);
                        if constexpr (PAIRED) {
                            const uint32_t at = next(walk);
                            if (i < NU || i < np) v[i] = lds_pk<T>(at);
                        } else {
                            const uint32_t at0 = next(walk), at1 = next(walk);
                            if (i < NU || i < np) v[i] = pk2(make_float2(lds_one<T>(at0), lds_one<T>(at1)));
                        }
                    }
#pragma unroll
                    for (int i = 0; i < NP; i += 2) {
                        m2 = max2(m2, upk2(v[i]));
                        m3 = max2(m3, upk2(v[i + 1]));
                    }
                    m = fmaxf(fmaxf(m2.x, m2.y), fmaxf(m3.x, m3.y));
                    if (odd) {
                        vt = to_f32(*last);
                        m = fmaxf(m, vt);
                    }
                }
                m = lanes_max(m, TPR, row_mask);
                const pk_t zero = psplat(0.f);
                float loss;
                if constexpr (KIND == kLSR) {
                    const float c2 = PAIRED ? kLog2e : exponent_scale(m), nm = -m * c2;
                    const pk_t l2e = psplat(c2), nml = psplat(nm);
                    pk_t ps[2] = {zero, zero}, px[2] = {zero, zero};
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        const pk_t x = x_of(i);
                        px[i & 1] = padd(px[i & 1], (i < NU || i < np) ? x : zero);
                        const pk_t e = pex2(pfma(x, l2e, nml));       // (0 past the end)
                        if constexpr (BWD) v[i] = e;                  // e^{x-m} takes x's place
                        ps[i & 1] = padd(ps[i & 1], e);
                    }
                    const float2 s2 = upk2(padd(ps[0], ps[1])), x2 = upk2(padd(px[0], px[1]));
                    float sum = s2.x + s2.y, sx = x2.x + x2.y;
                    if (odd) {
                        sx += vt;
                        vt = ex2f(fmaf(vt, c2, nm));
                        sum += vt;
                    }
                    for (int o = TPR >> 1; o > 0; o >>= 1) {
                        sum += __shfl_xor_sync(row_mask, sum, o);
                        sx += __shfl_xor_sync(row_mask, sx, o);
                    }
                    loss = kc.sumy * (m + __logf(sum)) - kc.lb_neg * sx - (kc.lb_pos - kc.lb_neg) * xl;
                    if constexpr (BWD) {
                        const float psc = prm.grad_mode == 2 ? gscale * to_f32(up) : gscale;
                        // g = (sumy e / s - lb_neg) scale; the target's lb_neg -> lb_pos
                        const float a = kc.sumy * __fdividef(psc, sum), b = -kc.lb_neg * psc;
                        const pk_t pa = psplat(a), pb = psplat(b);
                        Walk walk = begin();
#pragma unroll
                        for (int i = 0; i < NP; ++i) put(walk, i, pfma(v[i], pa, pb));
                        if (odd) *last = from_f32<T>(fmaf(vt, a, b));
                        if (owner) rp[lbi] = from_f32<T>(fmaf(ex2f(PAIRED ? fmaf(xl, kLog2e, nm) : (xl - m) * kLog2e), a, -kc.lb_pos * psc));
                    }
                } else {
                    const pk_t l2e = psplat(kLog2e), pnegm = psplat(-m);
                    pk_t ps[2] = {zero, zero}, psde[2] = {zero, zero}, psd[2] = {zero, zero};
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        const bool mine = i < NU || i < np;
                        // (past the end: 0 by choice, the row's maximum may be the lowest value too)
                        const pk_t d = mine ? padd(x_of(i), pnegm) : zero;
                        psd[i & 1] = padd(psd[i & 1], d);
                        if constexpr (!kHold) v[i] = d;               // d = x - m' takes x's place
                        const pk_t e = mine ? pex2(pmul(d, l2e)) : zero;
                        ps[i & 1] = padd(ps[i & 1], e);
                        psde[i & 1] = pfma(d, e, psde[i & 1]);
                    }
                    const float2 s2 = upk2(padd(ps[0], ps[1])), d2 = upk2(padd(psde[0], psde[1]));
                    const float2 x2 = upk2(padd(psd[0], psd[1]));
                    float sum = s2.x + s2.y, sde = d2.x + d2.y, sd = x2.x + x2.y;
                    if (odd) {
                        vt -= m;
                        sd += vt;
                        const float e = ex2f(vt * kLog2e);
                        sum += e;
                        sde = fmaf(vt, e, sde);
                    }
                    for (int o = TPR >> 1; o > 0; o >>= 1) {
                        sum += __shfl_xor_sync(row_mask, sum, o);
                        sde += __shfl_xor_sync(row_mask, sde, o);
                        sd += __shfl_xor_sync(row_mask, sd, o);
                    }
                    MarginRow fin;
                    fin.finish(m, sum, sde, sd, xl, xd, lbi, kc);
                    loss = fin.loss;
                    if constexpr (BWD) {
                        const float psc = prm.grad_mode == 2 ? gscale * to_f32(up) : gscale;
                        const float ca = (fin.r + kc.half_lam * (1.f - fin.sqx)) * psc, cb = kc.half_lam * psc;
                        const float cc = -kc.half_lam * kc.a * psc;
                        const pk_t pa = psplat(ca), pb = psplat(cb), pc = psplat(cc), pq = psplat(fin.inv_s);
                        Walk walk = begin();
#pragma unroll
                        for (int i = 0; i < NP; ++i) {
                            // (opaque: convert again instead of holding the first sweep's d in registers)
                            if constexpr (kHold) asm volatile("" : "+r"(held[i]));
                            const pk_t d = kHold ? padd(x_of(i), pnegm) : v[i];
                            const pk_t q = pmul(pex2(pmul(d, l2e)), pq);
                            put(walk, i, pfma(q, pfma(pb, d, pa), pc));
                        }
                        if (odd) {
                            const float q = ex2f(vt * kLog2e) * fin.inv_s;
                            *last = from_f32<T>(fmaf(q, fmaf(cb, vt, ca), cc));
                        }
                        if (owner) rp[lbi] = from_f32<T>(-fin.r * psc);
                    }
                }
                if (t == 0) {
                    if (!BWD && losses) losses[row] = from_f32<T>(loss);
                    acc_loss += double(loss);
                    ++acc_cnt;
                }
            }
            if (!BWD) {
                // (the stand-ins were plain stores: order them before the copy that refills the stage)
                if (KIND == kLMargin) fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars.empty[s]);
            } else {
                if (ragged) {
                    compute_sync(kShortCompute);
                    T *dst = static_cast<T *>(prm.grads) + row0 * C;
                    for (int e = tid; e < nrows * C; e += kShortCompute) dst[e] = tile[e];
                } else {
                    fence_proxy_async_smem();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars.ready[s]);
            }
        }
    }
    if (reduce) grid_reduce_finish(acc_loss, double(acc_cnt), prm.workspace, prm.out, sh_red, kTagSum, prm.defer != 0);
}

// -------------------------------------------------------------------------------------- rows_vec
// One 16-byte vector as pairs, and back.
template <typename T> struct VecPairs;
template <> struct VecPairs<float> {
    static constexpr int N = 2;
    static __device__ __forceinline__ void unpack(const uint4 &r, pk_t *p) {
        p[0] = pk2(make_float2(__uint_as_float(r.x), __uint_as_float(r.y)));
        p[1] = pk2(make_float2(__uint_as_float(r.z), __uint_as_float(r.w)));
    }
    static __device__ __forceinline__ uint4 pack(const pk_t *p) {
        const float2 a = upk2(p[0]), b = upk2(p[1]);
        return make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
    }
    static __device__ __forceinline__ float get(const uint4 &r, int e) {
        return __uint_as_float(e & 2 ? (e & 1 ? r.w : r.z) : (e & 1 ? r.y : r.x));
    }
    static __device__ __forceinline__ void put(uint4 &r, int e, float v) {
        const unsigned u = __float_as_uint(v);
        if (e == 0) r.x = u;
        if (e == 1) r.y = u;
        if (e == 2) r.z = u;
        if (e == 3) r.w = u;
    }
};
template <typename T, typename T2> struct VecPairs16 {
    static constexpr int N = 4;
    static __device__ __forceinline__ pk_t pair(unsigned w) { return ld_pk(reinterpret_cast<const T *>(&w)); }
    static __device__ __forceinline__ unsigned word(pk_t p) {
        unsigned w;
        st_pk(reinterpret_cast<T *>(&w), p);
        return w;
    }
    static __device__ __forceinline__ void unpack(const uint4 &r, pk_t *p) {
        p[0] = pair(r.x);
        p[1] = pair(r.y);
        p[2] = pair(r.z);
        p[3] = pair(r.w);
    }
    static __device__ __forceinline__ uint4 pack(const pk_t *p) {
        return make_uint4(word(p[0]), word(p[1]), word(p[2]), word(p[3]));
    }
    static __device__ __forceinline__ float get(const uint4 &r, int e) {
        const unsigned w = e & 4 ? (e & 2 ? r.w : r.z) : (e & 2 ? r.y : r.x);
        const float2 v = upk2(pair(w));
        return e & 1 ? v.y : v.x;
    }
    static __device__ __forceinline__ void put(uint4 &r, int e, float v) {
        const unsigned keep = e & 1 ? 0x0000ffffu : 0xffff0000u;
        const unsigned bits = word(psplat(v)) & ~keep;
        if ((e >> 1) == 0) r.x = (r.x & keep) | bits;
        if ((e >> 1) == 1) r.y = (r.y & keep) | bits;
        if ((e >> 1) == 2) r.z = (r.z & keep) | bits;
        if ((e >> 1) == 3) r.w = (r.w & keep) | bits;
    }
};
template <> struct VecPairs<__half> : VecPairs16<__half, __half2> {};
template <> struct VecPairs<__nv_bfloat16> : VecPairs16<__nv_bfloat16, __nv_bfloat162> {};

// NV: 16-byte vectors a lane can hold.
template <typename T, int KIND, bool BWD, int NV> constexpr int vec_blocks() {   // blocks per SM (registers)
    // (16-bit large-margin step, 1000 classes: 152 bytes spilled with three, 26.6 us; 24.1 us with two)
    if (KIND == kLMargin && BWD && sizeof(T) == 2 && NV == 4) return 2;
    return NV <= 4 ? 3 : 2;
}
// Vectors every lane holds for sure (launch_rows_vec picks the smallest NV of 8, 16, 32, 40, 48, 64 elements that
// holds a row): no check on those.
template <typename T, int NV> constexpr int vec_sure() {
    constexpr int n = NV * (16 / int(sizeof(T)));
    return (n == 64 ? 48 : n == 48 ? 40 : n == 40 ? 32 : n == 32 ? 16 : n == 16 ? 8 : 0) / (16 / int(sizeof(T)));
}
template <typename T, int KIND, bool BWD, int NV>
__global__ void __launch_bounds__(kVecThreads, vec_blocks<T, KIND, BWD, NV>())
rows_vec_kernel(const SoftmaxParams prm) {
    __shared__ double sh_red[64];
    using VP = VecPairs<T>;
    constexpr int VE = 16 / int(sizeof(T)), PV = VP::N;      // elements and pairs of a vector
    // the next row's vectors in flight under this row's arithmetic, where the registers hold both (float32 large margin
    // at 40 elements spills: [16384, 1100] step 39.6 us with, 33.3 us without)
    constexpr bool kAhead = NV * VE <= (KIND == kLMargin && sizeof(T) == 4 ? 32 : 40);
    // large margin replaces an element of the row below, which wants the vectors as loaded
    constexpr bool kRaw = kAhead || KIND == kLMargin;
    // accumulation chains: long rows wait on one chain's latency (float32 [32768, 2048] step 100 -> 95 us
    // with more), shorter ones want the registers ([65536, 1000] bfloat16 55 -> 61 us with two)
    constexpr int kChains = kRaw ? 1 : 4;
    const int lane = threadIdx.x & 31;
    const int C = prm.k.C, nvec = C / VE;
    const int cnt = (nvec - lane + 31) >> 5;                 // my vectors: lane, lane + 32, ...
    constexpr int NU = vec_sure<T, NV>();
    const int warps_b = int(blockDim.x) >> 5;
    const int64_t warps = int64_t(gridDim.x) * warps_b;
    const bool reduce = prm.out != nullptr;
    const T *gout = static_cast<const T *>(prm.grad_out);
    T *losses = static_cast<T *>(prm.losses);
    const LossConsts kc = prm.k;
    double acc_loss = 0.0, acc_cnt = 0.0;
    int64_t r = int64_t(blockIdx.x) * warps_b + (threadIdx.x >> 5);
    uint4 raw[NV];
    int64_t lb_next = 0;
    float up_next = 1.f;
    pk_t v[NV * PV];
    auto fetch = [&](int64_t row) {
        const uint4 *xr = static_cast<const uint4 *>(prm.logits) + row * nvec + lane;
        lb_next = __ldg(prm.labels + row);
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (i < NU || i < cnt) {
                if constexpr (kRaw) raw[i] = __ldcs(xr + 32 * i);
                else VP::unpack(__ldcs(xr + 32 * i), v + i * PV);
            }
        if (BWD && prm.grad_mode == 2) up_next = to_f32(gout[row]);
    };
    if (kAhead && r < prm.N) fetch(r);
    if (BWD && reduce) pdl_wait();                           // the divisor comes from the label count in front
    float gscale = 1.f;
    if (BWD) gscale = uniform_grad_scale(prm.grad_out, prm.grad_mode, prm.denom);
    for (; r < prm.N; r += warps) {
        if (!kAhead) fetch(r);
        const int64_t lb = lb_next;
        const float psc = (BWD && prm.grad_mode == 2) ? gscale * up_next : gscale;
        const bool valid = lb != prm.ignore;
        // (a label outside [0, C) that is not the ignore value is undefined in the reference: no target term here)
        const int lbi = (valid && lb >= 0 && lb < C) ? int(lb) : -1;
        float xl = 0.f, xd = 0.f;
        const int lvec = lbi / VE, le = lbi % VE;
        if (!kRaw && lbi >= 0) {                             // (uniform over the warp) in flight with the vectors
            const T *xs = static_cast<const T *>(prm.logits) + r * C;
            xl = to_f32(xs[lbi]);
        } else if (lbi >= 0) {
            if constexpr (KIND == kLMargin) {
                const float x0 = VP::get(raw[0], lbi == 0 ? 1 : 0), x1 = VP::get(raw[0], lbi <= 1 ? 2 : 1);
                xd = __shfl_sync(0xffffffffu, fmaxf(x0, x1), 0);
            }
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (lane + 32 * i == lvec) {
                    xl = VP::get(raw[i], le);
                    // large margin: the target's place holds another channel's logit during the sums
                    if constexpr (KIND == kLMargin) VP::put(raw[i], le, xd);
                }
            xl = __shfl_sync(0xffffffffu, xl, lvec & 31);
        } else if (KIND == kLMargin) {
            xl = kNegInf;
        }
        if constexpr (kRaw) {
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (i < NU || i < cnt) VP::unpack(raw[i], v + i * PV);
        }
        uint4 *grow = static_cast<uint4 *>(prm.grads) + r * nvec + lane;
        const int64_t row = r;
        if (kAhead && r + warps < prm.N) fetch(r + warps);
        if (!valid) {
            if (!BWD && losses && lane == 0) losses[row] = from_f32<T>(0.f);
            if (BWD) {
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    if (i < NU || i < cnt) __stcs(grow + 32 * i, make_uint4(0u, 0u, 0u, 0u));
            }
            continue;
        }
        float2 m2[kChains];
#pragma unroll
        for (int q = 0; q < kChains; ++q) m2[q] = splat2(kNegInf);
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (i < NU || i < cnt) {
#pragma unroll
                for (int p = 0; p < PV; ++p) {
                    float2 &mq = m2[(i * PV + p) % kChains];
                    mq = max2(mq, upk2(v[i * PV + p]));
                }
            }
#pragma unroll
        for (int q = 1; q < kChains; ++q) m2[0] = max2(m2[0], m2[q]);
        const float m = lanes_max(fmaxf(m2[0].x, m2[0].y), 32, 0xffffffffu);
        const pk_t zero = psplat(0.f);
        float loss;
        if constexpr (KIND == kLSR) {
            const float nm = -m * kLog2e;
            const pk_t l2e = psplat(kLog2e), nml = psplat(nm);
            pk_t ps[kChains], px[kChains];
#pragma unroll
            for (int q = 0; q < kChains; ++q) ps[q] = px[q] = zero;
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (i < NU || i < cnt) {
#pragma unroll
                    for (int p = 0; p < PV; ++p) {
                        pk_t &x = v[i * PV + p];
                        pk_t &pxq = px[(i * PV + p) % kChains], &psq = ps[(i * PV + p) % kChains];
                        pxq = padd(pxq, x);
                        x = pex2(pfma(x, l2e, nml));         // e^{x-m} takes x's place
                        psq = padd(psq, x);
                    }
                }
#pragma unroll
            for (int q = 1; q < kChains; ++q) {
                ps[0] = padd(ps[0], ps[q]);
                px[0] = padd(px[0], px[q]);
            }
            const float2 s2 = upk2(ps[0]), x2 = upk2(px[0]);
            const float sum = lanes_sum(s2.x + s2.y, 32, 0xffffffffu), sx = lanes_sum(x2.x + x2.y, 32, 0xffffffffu);
            loss = kc.sumy * (m + __logf(sum)) - kc.lb_neg * sx - (kc.lb_pos - kc.lb_neg) * xl;
            if constexpr (BWD) {
                const float a = kc.sumy * __fdividef(psc, sum), b = -kc.lb_neg * psc;
                const pk_t pa = psplat(a), pb = psplat(b);
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    if (i < NU || i < cnt) {
                        pk_t g[PV];
#pragma unroll
                        for (int p = 0; p < PV; ++p) g[p] = pfma(v[i * PV + p], pa, pb);
                        __stcs(grow + 32 * i, VP::pack(g));
                    }
                // target: (sumy e_l / s - lb_pos) scale, by the lane whose vector store covers it (program order)
                if (lbi >= 0 && ((lbi / VE) & 31) == lane)
                    (static_cast<T *>(prm.grads) + row * C)[lbi] =
                        from_f32<T>(fmaf(ex2f(fmaf(xl, kLog2e, nm)), a, -kc.lb_pos * psc));
            }
        } else {
            const pk_t l2e = psplat(kLog2e), pnegm = psplat(-m);
            pk_t ps = zero, psde = zero, psd = zero;
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (i < NU || i < cnt) {
#pragma unroll
                    for (int p = 0; p < PV; ++p) {
                        pk_t &x = v[i * PV + p];
                        x = padd(x, pnegm);                  // d = x - m' takes x's place
                        psd = padd(psd, x);
                        const pk_t e = pex2(pmul(x, l2e));
                        ps = padd(ps, e);
                        psde = pfma(x, e, psde);
                    }
                }
            const float2 s2 = upk2(ps), d2 = upk2(psde), x2 = upk2(psd);
            const float sum = lanes_sum(s2.x + s2.y, 32, 0xffffffffu), sde = lanes_sum(d2.x + d2.y, 32, 0xffffffffu);
            const float sd = lanes_sum(x2.x + x2.y, 32, 0xffffffffu);
            MarginRow fin;
            fin.finish(m, sum, sde, sd, xl, xd, lbi, kc);
            loss = fin.loss;
            if constexpr (BWD) {
                const pk_t pa = psplat((fin.r + kc.half_lam * (1.f - fin.sqx)) * psc), pb = psplat(kc.half_lam * psc);
                const pk_t pc = psplat(-kc.half_lam * kc.a * psc), pq = psplat(fin.inv_s);
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    if (i < NU || i < cnt) {
                        pk_t g[PV];
#pragma unroll
                        for (int p = 0; p < PV; ++p) {
                            const pk_t d = v[i * PV + p];
                            g[p] = pfma(pmul(pex2(pmul(d, l2e)), pq), pfma(pb, d, pa), pc);
                        }
                        __stcs(grow + 32 * i, VP::pack(g));
                    }
                if (lbi >= 0 && ((lbi / VE) & 31) == lane)
                    (static_cast<T *>(prm.grads) + row * C)[lbi] = from_f32<T>(-fin.r * psc);
            }
        }
        if (lane == 0) {
            if (!BWD && losses) losses[row] = from_f32<T>(loss);
            acc_loss += double(loss);
            acc_cnt += 1.0;
        }
    }
    if (reduce) grid_reduce_finish(acc_loss, acc_cnt, prm.workspace, prm.out, sh_red, kTagSum, prm.defer != 0);
}

// ----------------------------------------------------------------------------------- host side
template <typename T, int KIND, bool BWD> int launch_rows_vec(const SoftmaxParams &prm, cudaStream_t stream) {
    constexpr int VE = 16 / int(sizeof(T));
    const int nv = int((prm.C / VE + 31) / 32);
    const bool dep = BWD && prm.out && prm.after_count;
    // few rows: one warp per block first, so that they spread over the SMs
    const int64_t spread = (prm.N + sm_count() - 1) / sm_count();
    const int warps = int(spread < kVecWarps ? spread : kVecWarps);
    int64_t grid = (prm.N + warps - 1) / warps;
    auto go = [&](auto kern, int per_sm) {
        const int64_t cap = int64_t(sm_count()) * per_sm;    // all blocks resident: one reduction barrier per block
        if (grid > cap) grid = cap;
        launch_kernel(kern, dim3(unsigned(grid)), dim3(32 * warps), 0, stream, dep, prm);
    };
    constexpr int kSmall = sizeof(T) == 4 ? 8 : 4;           // 32 elements a lane
    if (nv <= kSmall / 4) go(rows_vec_kernel<T, KIND, BWD, kSmall / 4>, vec_blocks<T, KIND, BWD, kSmall / 4>());
    else if (nv <= kSmall / 2) go(rows_vec_kernel<T, KIND, BWD, kSmall / 2>, vec_blocks<T, KIND, BWD, kSmall / 2>());
    else if (nv <= kSmall) go(rows_vec_kernel<T, KIND, BWD, kSmall>, vec_blocks<T, KIND, BWD, kSmall>());
    else if (nv <= kSmall * 5 / 4) go(rows_vec_kernel<T, KIND, BWD, kSmall * 5 / 4>, vec_blocks<T, KIND, BWD, kSmall * 5 / 4>());
    else if (nv <= kSmall * 3 / 2) go(rows_vec_kernel<T, KIND, BWD, kSmall * 3 / 2>, vec_blocks<T, KIND, BWD, kSmall * 3 / 2>());
    else go(rows_vec_kernel<T, KIND, BWD, 2 * kSmall>, vec_blocks<T, KIND, BWD, 2 * kSmall>());
    return launch_status("softmax resident rows kernel launch");
}

template <typename T, int KIND, bool BWD, int MODE>
int launch_rows_short(SoftmaxParams prm, int tpr, cudaStream_t stream) {
    constexpr bool PAIRED = MODE != kSingles;
    const int units = int(PAIRED ? prm.C / 2 : prm.C);
    const int per_pair = PAIRED ? 1 : 2;
    const int np = ((units + tpr - 1) / tpr + per_pair - 1) / per_pair;
    prm.KS = tpr;
    const int R = kShortCompute / tpr;
    const size_t row_bytes = size_t(prm.C) * sizeof(T);
    // a stage of about 16 KB: several groups of rows where the rows are tiny
    int G = int(size_t(16384) / (size_t(R) * row_bytes));
    G = G < 1 ? 1 : G > 8 ? 8 : G;
    while (G > 1 && int64_t(R) * G * sm_count() * 3 > prm.N) G >>= 1;      // small inputs: all SMs first
    prm.rows = G;
    const size_t label_off = (size_t(R) * G * row_bytes + 127) & ~size_t(127);
    const size_t stage_bytes = label_off + size_t(R) * G * sizeof(int64_t);
    prm.stages = (BWD && stage_bytes <= size_t(36) * 1024) ? 3 : 2;
    const size_t smem = 128 + size_t(prm.stages) * stage_bytes;
    const int64_t n_stages = (prm.N + int64_t(R) * G - 1) / (int64_t(R) * G);
    const bool dep = BWD && prm.out && prm.after_count;
    int rc = B200_OK;
    auto go = [&](auto kern, int blocks) {                   // all blocks resident (registers, shared memory)
        int per_sm = int((224 * 1024) / (smem + 2048));
        if (per_sm > blocks) per_sm = blocks;
        if (per_sm < 1) per_sm = 1;
        int64_t grid = int64_t(sm_count()) * per_sm;
        if (grid > n_stages) grid = n_stages;
        if ((rc = set_smem(kern, smem)) != B200_OK) return;
        launch_kernel(kern, dim3(unsigned(grid)), dim3(kShortBlock), smem, stream, dep, prm);
    };
    if (np <= 4) go(rows_short_kernel<T, KIND, BWD, MODE, 4>, short_blocks<T, KIND, BWD, 4>());
    else if (np <= 8) go(rows_short_kernel<T, KIND, BWD, MODE, 8>, short_blocks<T, KIND, BWD, 8>());
    else if (np <= 10) go(rows_short_kernel<T, KIND, BWD, MODE, 10>, short_blocks<T, KIND, BWD, 10>());
    else if (np <= 12) go(rows_short_kernel<T, KIND, BWD, MODE, 12>, short_blocks<T, KIND, BWD, 12>());
    else if (np <= 16) go(rows_short_kernel<T, KIND, BWD, MODE, 16>, short_blocks<T, KIND, BWD, 16>());
    else if (MODE == kRotated || np <= 20) go(rows_short_kernel<T, KIND, BWD, MODE, 20>, short_blocks<T, KIND, BWD, 20>());
    else if constexpr (MODE != kRotated) go(rows_short_kernel<T, KIND, BWD, MODE, 32>, short_blocks<T, KIND, BWD, 32>());
    if (rc != B200_OK) return rc;
    return launch_status("softmax short-rows kernel launch");
}

template <typename T, int KIND, bool BWD> int launch_rows_typed(const SoftmaxParams &prm, cudaStream_t stream) {
    constexpr int VE = 16 / int(sizeof(T));
    // (labels that do not start on 16 bytes cannot be copied in bulk)
    if (prm.C % VE == 0 && (prm.C >= kVecMinC || (prm.C >= 16 * VE && !aligned16(prm.labels))))
        return launch_rows_vec<T, KIND, BWD>(prm, stream);
    // lanes per row: the fewest that keep a lane's share within 20 pairs (what a row costs besides its
    // elements is paid by every one of its lanes)
    int tpr = 1;
    while (tpr < 32 && (prm.C + tpr - 1) / tpr > 2 * kShortPairs) tpr <<= 1;
    // few rows: more lanes each while that brings more SMs to work and leaves a lane 8 channels
    while (tpr < 32 && prm.C / tpr >= 16 && prm.N * tpr < int64_t(kShortCompute) * sm_count()) tpr <<= 1;
    if (prm.C % 2 != 0) return launch_rows_short<T, KIND, BWD, kSingles>(prm, tpr, stream);
    if (prm.C % 4 == 0 && tpr <= 4) return launch_rows_short<T, KIND, BWD, kRotated>(prm, tpr, stream);
    return launch_rows_short<T, KIND, BWD, kPairs>(prm, tpr, stream);
}

template <int KIND, bool BWD> int launch_rows_dtype(int dtype, const SoftmaxParams &prm, cudaStream_t stream) {
    if (dtype == B200_F32) return launch_rows_typed<float, KIND, BWD>(prm, stream);
    if (dtype == B200_F16) return launch_rows_typed<__half, KIND, BWD>(prm, stream);
    if (dtype == B200_BF16) return launch_rows_typed<__nv_bfloat16, KIND, BWD>(prm, stream);
    set_error("unknown dtype code %d", dtype);
    return B200_ERR_ARG;
}

}  // namespace
}  // namespace b200

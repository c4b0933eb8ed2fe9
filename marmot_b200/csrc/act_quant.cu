// Activation quantizers: f32 rows -> Q8_K / Q8_0 values, bit-identical to the reference's
// matmul packers (src/backends/cpu/ops/matmul/quantized/matmul_quant_pack.c:23-62,106-169,
// scalar helpers src/backends/cpu/quantization/common/block.c:175-183,221-232).
#include "common.cuh"
#include "kernels.h"

#include <float.h>

namespace mcu {

// round-to-nearest-even through the 1.5*2^23 bit trick, as cpu_quant_matmul_nearest_int
// (matmul_quant_pack.c:11-21)
__device__ __forceinline__ int nearest_int(float v) {
    v = fminf(fmaxf(v, -4194303.0f), 4194303.0f);
    const float shifted = __fadd_rn(v, 12582912.0f);
    return (__float_as_int(shifted) & 0x007fffff) - 0x00400000;
}

// One warp per (token, 256-value block).  Lane l owns values l, l+32, ..., l+224.
__global__ void __launch_bounds__(256)
quantize_q8_k_kernel(const float *__restrict__ x, int ldx, int T, int K, int nb, int8_t *__restrict__ qs,
                     float *__restrict__ dq, int16_t *__restrict__ bsums, __half *__restrict__ xh) {
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= T * nb) return;
    const int t = w / nb, blk = w - t * nb;
    const float *row = x + (size_t)t * ldx + (size_t)blk * QK_K;
    const int len = min(QK_K, K - blk * QK_K);

    float v[8];
    float best_abs = 0.0f, best_val = 0.0f;
    int best_idx = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int idx = lane + 32 * i;
        v[i] = idx < len ? row[idx] : 0.0f;
        const float a = fabsf(v[i]);
        if (a > best_abs) {  // strict: the first occurrence wins
            best_abs = a;
            best_val = v[i];
            best_idx = idx;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, best_abs, o);
        const float ov = __shfl_xor_sync(0xffffffffu, best_val, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_idx, o);
        if (oa > best_abs || (oa == best_abs && oi < best_idx)) {
            best_abs = oa;
            best_val = ov;
            best_idx = oi;
        }
    }
    int8_t *qrow = qs + (size_t)t * nb * QK_K + (size_t)blk * QK_K;
    int16_t *brow = bsums + ((size_t)t * nb + blk) * 16;
    __half *hrow = xh != nullptr ? xh + (size_t)t * nb * QK_K + (size_t)blk * QK_K : nullptr;
    if (!(best_abs > 0.0f)) {
        // all-zero block: d = 0, zero quants (matmul_quant_pack.c:121-126)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            qrow[(i & 1) * 128 + (i >> 1) * 32 + lane] = 0;
            if (hrow != nullptr) hrow[lane + 32 * i] = __float2half_rn(0.0f);
        }
        if (lane < 16) brow[lane] = 0;
        if (lane == 0) dq[(size_t)t * nb + blk] = 0.0f;
        return;
    }
    const float iscale = __fdiv_rn(-127.0f, best_val);
    const float d = __fdiv_rn(1.0f, iscale);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int q = nearest_int(__fmul_rn(iscale, v[i]));
        q = min(q, 127);
        qrow[(i & 1) * 128 + (i >> 1) * 32 + lane] = (int8_t)q;
        if (hrow != nullptr) hrow[lane + 32 * i] = __float2half_rn(__fmul_rn(d, (float)q));
        // sums over 16 consecutive values: the 16 lanes of a half warp
        int s = q;
        s += __shfl_xor_sync(0xffffffffu, s, 8);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if ((lane & 15) == 0) brow[2 * i + (lane >> 4)] = (int16_t)s;
    }
    if (lane == 0) dq[(size_t)t * nb + blk] = d;
}

// One warp per (token, 32-value block); lane = value.
__global__ void __launch_bounds__(256)
quantize_q8_0_kernel(const float *__restrict__ x, int ldx, int T, int K, int nb, int8_t *__restrict__ qs,
                     float *__restrict__ dq, __half *__restrict__ xh) {
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const long total = (long)T * nb;
    for (long w = (long)blockIdx.x * wpb + (threadIdx.x >> 5); w < total; w += (long)gridDim.x * wpb) {
        const int t = (int)(w / nb), blk = (int)(w - (long)t * nb);
        const int k = blk * Q8_0_VALUES + lane;
        const float v = k < K ? x[(size_t)t * ldx + k] : 0.0f;
        float amax = fabsf(v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        float scale = __fdiv_rn(amax, 127.0f);
        if (scale < FLT_MIN) scale = 1.0f;
        const float inv = __fdiv_rn(1.0f, scale);
        int q = (int)roundf(__fmul_rn(v, inv));
        q = max(-127, min(127, q));
        const float d_stored = __half2float(__float2half_rn(scale));
        qs[(size_t)t * nb * Q8_0_VALUES + k] = (int8_t)q;
        if (xh != nullptr) xh[(size_t)t * nb * Q8_0_VALUES + k] = __float2half_rn(__fmul_rn(d_stored, (float)q));
        if (lane == 0) dq[(size_t)t * nb + blk] = d_stored;
    }
}

// Which value of a row goes to position k: every four consecutive values are stored as (0, 2, 1, 3) (see kernels.h).
__device__ __forceinline__ constexpr int act_order_source(int k) { return (k & ~3) | ((k & 1) << 1) | ((k >> 1) & 1); }

// fp16 operands for the tensor-core path: xh[t][k] = (d*q) * 2^-e_t, with one exponent per token chosen so
// that the largest magnitude of the row is about 2^14.  The power-of-two scale is exact, keeps large
// activations inside the fp16 range (and tiny ones out of the subnormals); the matmul epilogue multiplies
// the row back by rowscale[t] = 2^e_t.  One CTA per token.
__global__ void __launch_bounds__(256)
half_acts_kernel(int kq, const int8_t *__restrict__ qs, const float *__restrict__ dq, int nb, int kp,
                 __half *__restrict__ xh, float *__restrict__ rowscale) {
    __shared__ float red[8];
    __shared__ float inv_s;
    const int t = blockIdx.x;
    const float *drow = dq + (size_t)t * nb;
    float m = 0.0f;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) m = fmaxf(m, fabsf(drow[b]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float mm = 0.0f;
        for (int i = 0; i < 8; ++i) mm = fmaxf(mm, red[i]);
        mm *= 127.0f;  // bound of |d*q| over the row
        int e = 0;
        if (mm > 0.0f && mm < 3.0e38f) {
            (void)frexpf(mm, &e);  // mm = f * 2^e, f in [0.5, 1)
            e -= 14;
            e = max(-100, min(100, e));
        }
        inv_s = ldexpf(1.0f, -e);
        rowscale[t] = ldexpf(1.0f, e);
    }
    __syncthreads();
    const float inv = inv_s;
    const int8_t *qrow = qs + (size_t)t * kp;
    __half *hrow = xh + (size_t)t * kp;
    const int bv = kq ? QK_K : Q8_0_VALUES;
    for (int k = threadIdx.x; k < kp; k += blockDim.x) {
        const int src = act_order_source(k);
        const int blk = src / bv;
        const int pos = kq ? blk * QK_K + q8k_split_pos(src - blk * QK_K) : src;
        hrow[k] = __float2half_rn(__fmul_rn(__fmul_rn(drow[blk], inv), (float)qrow[pos]));
    }
}

// Quantise-and-stage in one kernel for the tensor-core matmul, which needs neither the int8 values nor the block
// sums in global memory: one CTA per token quantises the row block by block exactly as the kernels above (values
// and scales kept in shared memory), then writes xh and rowscale exactly as half_acts_kernel.  Launched with
// programmatic stream serialization: everything before griddepcontrol.wait is independent of earlier kernels.
// Sixteen staged values from sixteen quantised ones.
__device__ __forceinline__ void stage_group16(const int8_t *q16, float sc, __half *dst) {
    const uint4 raw = *(const uint4 *)q16;
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    float f[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) f[j] = __fmul_rn(sc, (float)(int8_t)(w[j >> 2] >> (8 * (j & 3))));
    uint32_t o[8];
#pragma unroll
    for (int p2 = 0; p2 < 8; ++p2) {
        const __half2 h = __floats2half2_rn(f[act_order_source(2 * p2)], f[act_order_source(2 * p2 + 1)]);
        o[p2] = *(const uint32_t *)&h;
    }
    uint4 *d = (uint4 *)dst;
    d[0] = make_uint4(o[0], o[1], o[2], o[3]);
    d[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// Quantise row t (of the staged matrix) block by block, exactly as the kernels above: values to q_s, scales to d_s (shared
// memory).  False when the row is not this rank's.  (src.x_out may be x: neither is __restrict__.)
// OP: STAGE_PLAIN = the row as it is; STAGE_NORM = rms_norm(x + add) * w; STAGE_SILU = silu(x) * x2 with the fast exponential and
// division (relative error about 1e-6: the result is quantised to eight bits right here, three orders of magnitude coarser);
// STAGE_SILU_RN = the same with the separately rounded exponential and division of the stand-alone kernels; STAGE_GELU.
// What bounds these launches is the latency of their loads, so every loop issues all loads of its turn before the first
// operation on them: a division's slow path, or the test for a pointer, between two loads made each one a trip of its own
// (rows of 14336 values: SiLU of 32 21 -> 9 us, of 4096 208 -> 124, 4.7 TB/s; add + RMSNorm of 64 rows of 4096 14.6 -> 5.9).
enum { STAGE_PLAIN = 0, STAGE_SILU = 1, STAGE_GELU = 2, STAGE_SILU_RN = 3, STAGE_NORM = 4 };
constexpr int NORM_BATCH = 16;

template <bool KQ, int OP>
__device__ __forceinline__ bool quantize_row(const float *x, int ldx, const ActSource &src, int K, int nb, int t,
                                             int8_t *q_s, float *d_s, float *red, float &inv_s) {
    constexpr bool GLU = OP == STAGE_SILU || OP == STAGE_GELU || OP == STAGE_SILU_RN;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    if (src.row_lo != nullptr && (t < *src.row_lo || t >= *src.row_hi)) return false;  // not this rank's row
    const size_t row_off = (size_t)(src.row_index != nullptr ? src.row_index[t] : t) * ldx;
    // what is read: the row itself (norm: the sum, once it is stored), the other half of the GLU or what is added
    const float *row = x + row_off;
    const float *other = GLU ? src.x2 + row_off : nullptr;
    float *x_out = src.x_out != nullptr ? src.x_out + row_off : nullptr;
    float norm_inv = 1.0f;
    if constexpr (OP == STAGE_NORM) {
        other = src.add != nullptr ? src.add + row_off : nullptr;
        float sum = 0.0f;
        // (256 threads whatever the block: the order of the sum is that of the stand-alone kernel)
        for (int i0 = threadIdx.x; i0 < K && threadIdx.x < 256; i0 += 256 * NORM_BATCH) {
            float v[NORM_BATCH];
#pragma unroll
            for (int j = 0; j < NORM_BATCH; ++j) v[j] = i0 + 256 * j < K ? row[i0 + 256 * j] : 0.0f;
            if (other != nullptr) {
                float a[NORM_BATCH];
#pragma unroll
                for (int j = 0; j < NORM_BATCH; ++j) a[j] = i0 + 256 * j < K ? other[i0 + 256 * j] : 0.0f;
#pragma unroll
                for (int j = 0; j < NORM_BATCH; ++j) v[j] = __fadd_rn(v[j], a[j]);
            }
#pragma unroll
            for (int j = 0; j < NORM_BATCH; ++j) sum += v[j] * v[j];
            if (x_out != nullptr) {
#pragma unroll
                for (int j = 0; j < NORM_BATCH; ++j)
                    if (i0 + 256 * j < K) x_out[i0 + 256 * j] = v[j];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0 && warp < 8) red[warp] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            float s = 0.0f;
            for (int i = 0; i < 8; ++i) s += red[i];
            inv_s = __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(s, (float)K), src.eps)));
        }
        __syncthreads();
        norm_inv = inv_s;
        __syncthreads();  // red and inv_s are used again below
        if (x_out != nullptr) {  // the packer reads the sums back (other threads' elements too: all written before
            row = x_out;         // the barriers above) instead of adding again
            other = nullptr;
        }
    }
    // N values of a block, 32 apart: all loads, then the operations
    auto values = [&](int k0, auto &v) {
        constexpr int N = sizeof(v) / sizeof(v[0]);
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = k0 + 32 * i < K ? row[k0 + 32 * i] : 0.0f;
        if constexpr (OP == STAGE_PLAIN) return;
        float o[N];
        if (other != nullptr) {
#pragma unroll
            for (int i = 0; i < N; ++i) o[i] = k0 + 32 * i < K ? other[k0 + 32 * i] : 0.0f;
        }
        if constexpr (OP == STAGE_NORM) {
            float w[N];
            if (src.norm_w != nullptr) {
#pragma unroll
                for (int i = 0; i < N; ++i) w[i] = k0 + 32 * i < K ? src.norm_w[k0 + 32 * i] : 0.0f;
            }
            if (other != nullptr) {
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] = __fadd_rn(v[i], o[i]);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = __fmul_rn(v[i], norm_inv);
            if (src.norm_w != nullptr) {
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] = __fmul_rn(v[i], __fadd_rn(w[i], src.w_off));
            }
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const float g = v[i];
                float a;
                if constexpr (OP == STAGE_GELU) a = __fmul_rn(__fmul_rn(0.5f, g), __fadd_rn(1.0f, erff(__fmul_rn(g, 0.7071067811865475f))));
                else if constexpr (OP == STAGE_SILU_RN) a = __fdiv_rn(g, __fadd_rn(1.0f, expf(-g)));
                else a = __fdividef(g, __fadd_rn(1.0f, __expf(-g)));
                v[i] = __fmul_rn(a, o[i]);
            }
            if (KQ && x_out != nullptr) {
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (k0 + 32 * i < K) x_out[k0 + 32 * i] = v[i];
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (k0 + 32 * i >= K) v[i] = 0.0f;
    };
    if (KQ) {
        for (int blk = warp; blk < nb; blk += n_warps) {
            float v[8];
            values(blk * QK_K + lane, v);
            float best_abs = 0.0f, best_val = 0.0f;
            int best_idx = 0x7fffffff;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float a = fabsf(v[i]);
                if (a > best_abs) {
                    best_abs = a;
                    best_val = v[i];
                    best_idx = lane + 32 * i;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float oa = __shfl_xor_sync(0xffffffffu, best_abs, o);
                const float ov = __shfl_xor_sync(0xffffffffu, best_val, o);
                const int oi = __shfl_xor_sync(0xffffffffu, best_idx, o);
                if (oa > best_abs || (oa == best_abs && oi < best_idx)) {
                    best_abs = oa;
                    best_val = ov;
                    best_idx = oi;
                }
            }
            float d = 0.0f, iscale = 0.0f;
            if (best_abs > 0.0f) {
                iscale = __fdiv_rn(-127.0f, best_val);
                d = __fdiv_rn(1.0f, iscale);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                int q = best_abs > 0.0f ? min(nearest_int(__fmul_rn(iscale, v[i])), 127) : 0;
                q_s[blk * QK_K + lane + 32 * i] = (int8_t)q;
            }
            if (lane == 0) d_s[blk] = d;
        }
    } else {
        // four blocks in turn per warp, their loads together
        for (int blk0 = 4 * warp; blk0 < nb; blk0 += 4 * n_warps) {
            float v[4];
            values(blk0 * Q8_0_VALUES + lane, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int blk = blk0 + i;
                if (blk >= nb) break;
                float amax = fabsf(v[i]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                float scale = __fdiv_rn(amax, 127.0f);
                if (scale < FLT_MIN) scale = 1.0f;
                const float inv = __fdiv_rn(1.0f, scale);
                int q = (int)roundf(__fmul_rn(v[i], inv));
                q = max(-127, min(127, q));
                q_s[blk * Q8_0_VALUES + lane] = (int8_t)q;
                if (lane == 0) d_s[blk] = __half2float(__float2half_rn(scale));
            }
        }
    }
    return true;
}

// Lets the matmul behind start, and waits for the kernel ahead.  A grouped matmul reads the groups' counts before its own wait, so it may
// start only when the routing kernels are complete: this kernel's wait first.
__device__ __forceinline__ void stage_begin(const ActSource &src) {
    if (src.row_lo == nullptr) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (src.row_lo != nullptr) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Few rows: up to a thousand threads per row, so that a row is one or two trips to L2 (latency bounds the launch: 64 rows of
// 4096 values 3.3 us with 256 threads); many rows: 256 threads, and as many rows at a time.
template <bool KQ, int OP>
__global__ void __launch_bounds__(1024)
act_half_fused_kernel(const float *x, int ldx, ActSource src, int K, int nb, __half *__restrict__ xh,
                      float *__restrict__ rowscale) {
    extern __shared__ __align__(16) uint8_t act_sm[];
    constexpr int BV = KQ ? QK_K : Q8_0_VALUES;
    const int kp = nb * BV;
    int8_t *q_s = (int8_t *)act_sm;
    float *d_s = (float *)(act_sm + ((kp + 15) & ~15));
    __shared__ float red[32];
    __shared__ float inv_s;
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    stage_begin(src);
    if (!quantize_row<KQ, OP>(x, ldx, src, K, nb, t, q_s, d_s, red, inv_s)) return;
    __syncthreads();
    float m = 0.0f;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) m = fmaxf(m, fabsf(d_s[b]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float mm = 0.0f;
        for (int i = 0; i < n_warps; ++i) mm = fmaxf(mm, red[i]);
        mm *= 127.0f;
        int e = 0;
        if (mm > 0.0f && mm < 3.0e38f) {
            (void)frexpf(mm, &e);
            e -= 14;
            e = max(-100, min(100, e));
        }
        inv_s = ldexpf(1.0f, -e);
        rowscale[t] = ldexpf(1.0f, e);
    }
    __syncthreads();
    const float inv = inv_s;
    __half *hrow = xh + (size_t)t * kp;
    for (int g = threadIdx.x; g < kp / 16; g += blockDim.x) {
        const float sc = __fmul_rn(d_s[(16 * g) / BV], inv);
        stage_group16(q_s + 16 * g, sc, hrow + 16 * g);
    }
}

// The operands of the integer tensor-core matmul (gemm_ti.cu) for K-quants: per row and 256-value block 384 bytes, the 256
// quants, then the sums of its sub-blocks split as 64 * hi + lo into 8-bit values (lo from byte 256, hi from byte 288 on).
// SUB = 32 (Q4_K: eight sums) or 16 (Q6_K: sixteen sums, and two planes of quants, in which the even / the odd sub-blocks are
// zero: the matmul multiplies 32 values at a time and needs the sums of 16).  The block's scale follows at byte 320.
template <int SUB, int OP>
__global__ void __launch_bounds__(1024)
act_int_fused_kernel(const float *x, int ldx, ActSource src, int K, int nb, uint8_t *__restrict__ xq, size_t plane) {
    extern __shared__ __align__(16) uint8_t act_sm[];
    int8_t *q_s = (int8_t *)act_sm;
    float *d_s = (float *)(act_sm + nb * QK_K);
    __shared__ float red[32];
    __shared__ float inv_s;
    const int t = blockIdx.x;
    stage_begin(src);
    if (!quantize_row<true, OP>(x, ldx, src, K, nb, t, q_s, d_s, red, inv_s)) return;
    __syncthreads();
    uint8_t *row = xq + (size_t)t * nb * 384;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) *(float *)(row + b * 384 + 320) = d_s[b];
    constexpr int PER = SUB / 16;  // a sub-block per thread: one or two 16-byte words
    for (int g = threadIdx.x; g < nb * (QK_K / SUB); g += blockDim.x) {
        const int blk = g / (QK_K / SUB), at = g % (QK_K / SUB);
        uint8_t *o = row + blk * 384;
        int sum = 0;
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const uint4 v = *(const uint4 *)(q_s + SUB * g + 16 * n);
            sum = __dp4a((int)v.x, 0x01010101, __dp4a((int)v.y, 0x01010101, __dp4a((int)v.z, 0x01010101, __dp4a((int)v.w, 0x01010101, sum))));
            if (SUB == 16) {
                const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
                *(uint4 *)(o + 16 * at) = at & 1 ? zero : v;
                *(uint4 *)(o + plane + 16 * at) = at & 1 ? v : zero;
            } else {
                *(uint4 *)(o + SUB * at + 16 * n) = v;
            }
        }
        const int lo = sum & 63;
        o[256 + at] = (uint8_t)lo;
        o[288 + at] = (uint8_t)((sum - lo) >> 6);
        // the rest of the two 32-byte groups is zero
        constexpr int REST = 32 * SUB / QK_K - 1;  // per thread
#pragma unroll
        for (int n = 0; n < REST; ++n) o[256 + QK_K / SUB + REST * at + n] = o[288 + QK_K / SUB + REST * at + n] = 0;
    }
}

static int stage_op(const ActSource &src) {
    if (src.x2 != nullptr) return src.glu == 2 ? STAGE_GELU : src.glu == 3 ? STAGE_SILU_RN : STAGE_SILU;
    return src.norm ? STAGE_NORM : STAGE_PLAIN;
}

size_t act_half_fused_smem(int kind, int K) {
    const int bv = block_values(kind), nb = (K + bv - 1) / bv;
    return (size_t)((nb * bv + 15) & ~15) + (size_t)nb * sizeof(float);
}

cudaError_t launch_act_half_fused_from(int kind, const float *x, int ldx, const ActSource &src, int T, int K,
                                       __half *xh, float *rowscale, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    const int bv = block_values(kind), nb = (K + bv - 1) / bv;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)T, 1, 1);
    int warps = 8;
    if (T < 512) {
        const int want = kind != KIND_Q8_0 ? nb : nb / 4;  // a 256-value block, or four 32-value ones in turn, per warp
        // K-quants, more rows than SMs: registers allow 1024 threads on an SM, so two rows at a time on each, and beyond 296 rows 32 * SMs / T
        // warps a row: two rows at a time up to 430, three from there on, which is one wave from 431 to 444 rows and two elsewhere, the second one
        // short (whole calls, 32 warps and so: 180 x 14336 x 4096 Q6_K 35.5, 34.8 us, 300 50.9, 48.1, 400 Q4_K 55.0, 52.4; 500 x 4096 x 4096
        // 27.0, 26.4.  Rows of Q8_0 keep theirs: 300 x 4096 x 14336 46.9, 48.5).
        warps = want < 8 ? 8 : want > 32 ? 32 : want;
        if (kind != KIND_Q8_0 && T > 64 && warps > 8) {  // (else the count of SMs makes no difference)
            const int sms = device_sm_count(), most = T <= sms ? 32 : T <= 2 * sms ? 16 : 32 * sms / T;
            if (warps > most) warps = most < 8 ? 8 : most;
        }
    }
    cfg.blockDim = dim3((unsigned)(32 * warps), 1, 1);
    cfg.dynamicSmemBytes = act_half_fused_smem(kind, K);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool kq = kind != KIND_Q8_0;
#define MCU_STAGE(OP) \
    (kq ? cudaLaunchKernelEx(&cfg, act_half_fused_kernel<true, OP>, x, ldx, src, K, nb, xh, rowscale) \
        : cudaLaunchKernelEx(&cfg, act_half_fused_kernel<false, OP>, x, ldx, src, K, nb, xh, rowscale))
    switch (stage_op(src)) {
    case STAGE_SILU: return MCU_STAGE(STAGE_SILU);
    case STAGE_SILU_RN: return MCU_STAGE(STAGE_SILU_RN);
    case STAGE_GELU: return MCU_STAGE(STAGE_GELU);
    case STAGE_NORM: return MCU_STAGE(STAGE_NORM);
    default: return MCU_STAGE(STAGE_PLAIN);
    }
#undef MCU_STAGE
}

cudaError_t launch_act_int_fused(int kind, const float *x, int ldx, const ActSource &src, int rows, int K, uint8_t *xq, cudaStream_t s) {
    if (rows <= 0) return cudaSuccess;
    const int nb = (K + QK_K - 1) / QK_K;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows, 1, 1);
    cfg.blockDim = dim3((unsigned)(32 * (nb < 8 ? 8 : nb > 32 ? 32 : nb)), 1, 1);
    cfg.dynamicSmemBytes = act_half_fused_smem(kind, K);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const size_t plane = (size_t)rows * nb * 384;
    auto launch = [&](auto kernel) {
        if (cfg.dynamicSmemBytes > 48 * 1024)  // (rows of more than 48,000 values)
            if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ACT_INT_MAX_SMEM)) return e;
        return cudaLaunchKernelEx(&cfg, kernel, x, ldx, src, K, nb, xq, plane);
    };
#define MCU_STAGE(OP) (kind == KIND_Q6_K ? launch(act_int_fused_kernel<16, OP>) : launch(act_int_fused_kernel<32, OP>))
    switch (stage_op(src)) {
    case STAGE_SILU:
    case STAGE_SILU_RN: return MCU_STAGE(STAGE_SILU_RN);
    case STAGE_GELU: return MCU_STAGE(STAGE_GELU);
    case STAGE_NORM: return MCU_STAGE(STAGE_NORM);
    default: return MCU_STAGE(STAGE_PLAIN);
    }
#undef MCU_STAGE
}

cudaError_t launch_half_acts(int kind, const ActBuffers &a, int T, int K, __half *xh, float *rowscale, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    const int bv = block_values(kind), nb = (K + bv - 1) / bv;
    half_acts_kernel<<<T, 256, 0, s>>>(kind != KIND_Q8_0, a.qs, a.d, nb, nb * bv, xh, rowscale);
    return cudaGetLastError();
}

cudaError_t launch_quantize_act(int kind, const float *x, int ldx, int T, int K, const ActBuffers &a, __half *xh,
                                cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    if (kind == KIND_Q8_0) {
        const int nb = (K + Q8_0_VALUES - 1) / Q8_0_VALUES;
        const long warps = (long)T * nb;
        const int blocks = (int)min((warps + 7) / 8, (long)148 * 16);
        quantize_q8_0_kernel<<<blocks, 256, 0, s>>>(x, ldx, T, K, nb, a.qs, a.d, xh);
    } else {
        const int nb = (K + QK_K - 1) / QK_K;
        const long warps = (long)T * nb;
        quantize_q8_k_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(x, ldx, T, K, nb, a.qs, a.d, a.bsums, xh);
    }
    return cudaGetLastError();
}

}  // namespace mcu

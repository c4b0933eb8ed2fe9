// Quantized matmul on tcgen05 with the WEIGHTS in tensor memory: out[t][f] = sum_k xh[t][k] * W[f][k].
//
// What bounds this path is shared-memory bandwidth, not the tensor pipe or L2: a kernel that writes dequantised fp16 weight
// tiles to shared memory and lets the MMA read them back moves 32 KB per 128 x 64 weights that way alone (64 tokens: 58 KB per
// 64-wide K step = 450 cycles at 128 B per cycle, the step time such a kernel measured; the tensor pipe needs 128).  Here the
// converter threads put the dequantised values straight into tensor memory (tcgen05.st, one weight row per thread, no
// swizzle, no bank conflicts) and the MMA takes its A operand from there; shared memory carries the packed blocks and the
// activation tile only.
//
//   warps 0..15   converters: four groups of four warps; group g takes half g & 1 (one stage, 128 values of K) of the slabs
//                 j with j % 2 == g >> 1.  A warp owns the 32 TMEM lanes of its quadrant, a thread one weight row: packed words from shared memory,
//                 packed-half arithmetic, tcgen05.st.  The same warps run the epilogue.
//   warp 16       issues tcgen05.mma (M = 128, N = bn <= 256 tokens, K = 16) and tcgen05.commit
//   warp 17       activation tiles by TMA (128-byte swizzle)
//   warp 18       packed weight slabs (128 rows x 256 values) into a shared-memory ring, by TMA.  Rows that are not 16-byte
//                 multiples (Q6_K with K % 2048 != 0) come as eight copies of every eighth row: eight rows always are.
//
// Measured (whole mcu_linear call, graph replay, microseconds before -> now): Q4_K 64 x 4096 x 14336 31.0 -> 17.3,
// 17 x 4096 x 4096 13.2 -> 10.1, 64 x 4096 x 1024 17.2 -> 9.5, 2048 x 4096 x 14336 274 -> 213 (1127 TFLOP/s: 0.83 of the
// sustained cuBLAS rate, the clock is at the power limit); Q6_K 37 x 14336 x 4096 40.0 -> 25.4, 512 x 5632 x 2048 142 -> 29.0.
// Up to 128 tokens the converters bound a slab (Q4_K about 1100 cycles for 32768 weights in tiles of up to 64 tokens, 1500 in wider ones;
// instruction issue); from 256 on the MMAs run at their peak rate (2050 cycles per slab) and what is left is the epilogue (7500 cycles
// beside a tile's 33000 of MMAs, about half of them ahead of the next tile's).  Beside the kernel a call has its staging launch: of the 17 us at 64 x 4096 x 14336 it and the releases around it take 6.5.
//
// A CTA has one or several output tiles, or a cluster shares one along K and adds its shares up through distributed shared memory, or the slabs of
// all tiles are cut into equal ranges: a tile cut between CTAs is then summed from partial tiles by the one that draws the last
// ticket, in a fixed order; nobody waits for another CTA (kernels on several streams may share the device).  ts_spread chooses.
// Every mbarrier wait is bounded; no TMA multicast.
#include "common.cuh"
#include "gemm_ts_dev.cuh"
#include "kernels.h"
#include "tma_utils.cuh"

#include <cuda.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <type_traits>

namespace mcu {

constexpr int TS_STAGES = 4;    // = converter groups: group g owns stage slot g, so every barrier phase is seen in order
constexpr int TS_CONV = 16;     // converter warps
constexpr int TS_MMA_WARP = TS_CONV, TS_B_WARP = TS_CONV + 1, TS_W_WARP = TS_CONV + 2;
constexpr int TS_THREADS = (TS_W_WARP + 1) * 32;
constexpr int TS_D_COLS = 256;  // accumulator columns; the A ring (4 x 64 columns) follows

// D += A * B, A in tensor memory (two fp16 per 32-bit column), B in shared memory.
__device__ __forceinline__ void ts_mma(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
// ---- converters: 128 values of one weight row (half `n` of a 256-value slab) as 64 packed-half columns, K order (0, 2, 1, 3)
//      inside every group of four.  Everything is read from the slab first and the slab released (`done`),
//      so that its refill overlaps the arithmetic; `emit` gets the columns in four quarters (registers). ----

// Q4_K: the arithmetic keeps the 6-bit scales and the fp16 block scales in packed halves: d * sc and dmin * m are single
// fp16 roundings of exact products, and a weight is one HFMA2 of exact operands.
// (w & mask) | bits in one LOP3: left to itself the compiler takes two, with an immediate each, and the ALU pipe (a warp
// instruction every two cycles) is what bounds the converters.
__device__ __forceinline__ uint32_t ts_and_or(uint32_t w, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(bits));
    return r;
}
template <class Done, class Emit>
__device__ __forceinline__ void ts_conv_q4k(const uint8_t *rowp, int n, Done done, Emit emit) {
    const uint4 hdr = *(const uint4 *)rowp;  // d, dmin | scales[0..3] | scales[4..7] | scales[8..11]
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = *(const uint4 *)(rowp + 16 + 64 * n + 16 * i);
    done();
    uint32_t sc4, mn4;  // the four sub-blocks' 6-bit scales and mins, one per byte
    if (n == 0) {
        sc4 = hdr.y & 0x3F3F3F3Fu;
        mn4 = hdr.z & 0x3F3F3F3Fu;
    } else {
        sc4 = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
        mn4 = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
    }
    const __half2 k1024 = as_half2(0x64006400u), k64 = as_half2(0x54005400u);
    const __half2 dd = as_half2(__byte_perm(hdr.x, 0u, 0x1010));                // (d, d)
    const __half2 nd = as_half2(__byte_perm(hdr.x, 0u, 0x3232) ^ 0x80008000u);  // (-dmin, -dmin)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 q0 = q[2 * h], q1 = q[2 * h + 1];
        const uint32_t pick = h == 0 ? 0x4140u : 0x4342u;
        const __half2 s2 = __hmul2(__hsub2(as_half2(__byte_perm(sc4, 0x64646464u, pick)), k1024), dd);
        const __half2 m2 = __hmul2(__hsub2(as_half2(__byte_perm(mn4, 0x64646464u, pick)), k1024), nd);
        const __half2 sa = bcast_lo(s2), sb = bcast_hi(s2), ma = bcast_lo(m2), mb = bcast_hi(m2);
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        uint32_t o[16];
        // 0x6400 | v = 1024 + v;  0x5400 | (v << 4) = 64 + v
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const __half2 a0 = as_half2(ts_and_or(w[i], 0x000F000Fu, 0x64006400u)), a1 = as_half2(ts_and_or(w[i] >> 8, 0x000F000Fu, 0x64006400u));
            o[2 * i] = as_u32(__hfma2(__hsub2(a0, k1024), sa, ma));
            o[2 * i + 1] = as_u32(__hfma2(__hsub2(a1, k1024), sa, ma));
        }
        emit(2 * h, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const __half2 b0 = as_half2(ts_and_or(w[i], 0x00F000F0u, 0x54005400u)), b1 = as_half2(ts_and_or(w[i] >> 8, 0x00F000F0u, 0x54005400u));
            o[2 * i] = as_u32(__hfma2(__hsub2(b0, k64), sb, mb));
            o[2 * i + 1] = as_u32(__hfma2(__hsub2(b1, k64), sb, mb));
        }
        emit(2 * h + 1, o);
    }
}

// Q6_K: value 128 n + 32 c + l has its low four bits in byte 64 n + 32 (c & 1) + l of ql (high nibble for c >= 2), its high two
// in bits 2 c of byte 32 n + l of qh.  d * sc is rounded to fp16 before the product with the quant; ONCE: that product is formed in 32
// bits and rounded once (error of the result 2.9e-4 instead of 3.6e-4): rows that are not 16-byte multiples, which always had it.
// Such rows start anywhere; the others all at byte `phase` behind a 16-byte boundary.
template <bool ONCE, class Done, class Emit>
__device__ __forceinline__ void ts_conv_q6k(const uint8_t *blk, uint32_t phase, int n, Done done, Emit emit) {
    uint32_t ql[16], qh[8], sc[2];
    if (ONCE) {
        tm_lds_words<16>(blk + n * 64, ql);
        tm_lds_words<8>(blk + 128 + n * 32, qh);
    } else {
        ts_lds_phase<16>(blk - phase + n * 64, phase, ql);
        ts_lds_phase<8>(blk - phase + 128 + n * 32, phase, qh);
    }
    tm_lds_words<2>(blk + 192 + n * 8, sc);
    const float d = half_bits_to_float(*(const uint16_t *)(blk + 208));
    done();
    const __half2 off = as_half2(0x64206420u);  // 1024 + 32
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            uint32_t o[16];
            const int c = 2 * t + b;
            const uint32_t sw = sc[t] >> (16 * b);
            const float f0 = __fmul_rn(d, (float)(int8_t)sw), f1 = __fmul_rn(d, (float)(int8_t)(sw >> 8));  // (exact)
            const __half2 ds0 = __float2half2_rn(f0), ds1 = __float2half2_rn(f1);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t hi = 2 * c >= 4 ? qh[j] >> (2 * c - 4) : qh[j] << (4 - 2 * c);  // two bits at bit 4
                const uint32_t u = ((ql[8 * b + j] >> (4 * t)) & 0x0F0F0F0Fu) | (hi & 0x30303030u);
                __half2 v0, v1;
                bytes_to_half2(u, off, v0, v1);
                if (ONCE) {
                    const float f = j < 4 ? f0 : f1;
                    const float2 w0 = __half22float2(v0), w1 = __half22float2(v1);
                    o[2 * j] = as_u32(__floats2half2_rn(__fmul_rn(w0.x, f), __fmul_rn(w0.y, f)));
                    o[2 * j + 1] = as_u32(__floats2half2_rn(__fmul_rn(w1.x, f), __fmul_rn(w1.y, f)));
                    continue;
                }
                const __half2 ds = j < 4 ? ds0 : ds1;
                o[2 * j] = as_u32(__hmul2(v0, ds));
                o[2 * j + 1] = as_u32(__hmul2(v1, ds));
            }
            emit(c, o);
        }
    }
}

// Q8_0: blocks 4 n .. 4 n + 3 of the slab; blocks at or beyond `n_blk` (the end of the row) are zero.
__device__ __forceinline__ void ts_conv_q8_block(const uint32_t (&q)[8], uint32_t d_bits, uint32_t (&o)[16]) {
    const __half2 off = as_half2(0x64806480u);  // 1024 + 128
    const __half2 dh = as_half2(__byte_perm(d_bits, 0u, 0x1010));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        __half2 v0, v1;
        bytes_to_half2(q[j] ^ 0x80808080u, off, v0, v1);
        o[2 * j] = as_u32(__hmul2(v0, dh));
        o[2 * j + 1] = as_u32(__hmul2(v1, dh));
    }
}
// rows on 16-byte boundaries: a pair of blocks (68 bytes) lies in five 16-byte words at a known offset
template <int N, class Done, class Emit>
__device__ __forceinline__ void ts_conv_q8_0(const uint8_t *rowp, int n_blk, Done done, Emit emit) {
    constexpr int S0 = 136 * N;
    uint32_t w2[2][20];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const uint4 v = *(const uint4 *)(rowp + ((S0 + 68 * t) & ~15) + 16 * i);
            w2[t][4 * i] = v.x, w2[t][4 * i + 1] = v.y, w2[t][4 * i + 2] = v.z, w2[t][4 * i + 3] = v.w;
        }
    done();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const uint32_t (&w)[20] = w2[t];
        const int o4 = 2 * N + t;  // word offset of the pair inside its window
        uint32_t o[16], q[8];
        const int c = 4 * N + 2 * t;
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = __funnelshift_r(w[o4 + j], w[o4 + j + 1], 16);
        // (quants are finite whatever the bytes, so a zero scale clears a block)
        ts_conv_q8_block(q, c < n_blk ? w[o4] : 0u, o);
        emit(2 * t, o);
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = w[o4 + 9 + j];
        ts_conv_q8_block(q, c + 1 < n_blk ? w[o4 + 8] >> 16 : 0u, o);
        emit(2 * t + 1, o);
    }
}
template <class Done, class Emit>
__device__ __forceinline__ void ts_conv_q8_0_loose(const uint8_t *rowp, int n, int n_blk, Done done, Emit emit) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            uint32_t o[16];
            const int c = 4 * n + 2 * t + b;
            const uint8_t *blk = rowp + c * Q8_0_BYTES;
            uint32_t q[8];
            tm_lds_words<8>(blk + 2, q);
            ts_conv_q8_block(q, c < n_blk ? *(const uint16_t *)blk : 0u, o);
            if (2 * t + b == 3) done();
            emit(2 * t + b, o);
        }
    }
}

// Sixteen columns (tokens col0 ..) of this thread's weight row into the output; their scales are in the lanes from `src` on of
// `scale`.  (Scales read from memory between the stores, which may alias them, made the epilogue of a 256-column tile cost
// 7700 cycles; read per chunk ahead of its stores, still 7500: a trip to L2 each.)
__device__ __forceinline__ void ts_store16(float *outp, int ldo, int col0, int count, bool live, float bias, float scale, int src,
                                           const uint32_t (&v)[16]) {
    float *o = outp + (size_t)col0 * ldo;
#pragma unroll
    for (int jj = 0; jj < 16; ++jj) {
        const float sc = __shfl_sync(0xffffffffu, scale, src + jj);
        if (live && col0 + jj < count) *o = __uint_as_float(v[jj]) * sc + bias;
        o += ldo;
    }
}

// LOOSE: the weight rows are not 16-byte multiples.  (A branch in the kernel costs the aligned rows registers, in Q6_K most: 256
// routes to 8 experts of 3 x 14336 x 4096 499 us, 461 so.)
template <int KIND, bool LOOSE>
__global__ void __launch_bounds__(TS_THREADS, 1)
gemm_ts_kernel(const __grid_constant__ TsMaps maps, const __grid_constant__ TsParams p) {
    extern __shared__ uint8_t smem_raw[];
    using SL = TsSlab<KIND>;
    constexpr bool loose = LOOSE;
    constexpr uint32_t SLAB = ts_slab_bytes<KIND>(LOOSE);
    constexpr uint32_t S = TS_STAGES;
    const uint32_t raw_addr = tm_smem_u32(smem_raw);
    const uint32_t bar_base = (raw_addr + 15u) & ~15u;
    const uint32_t tile_base = (bar_base + 512u + 1023u) & ~1023u;
    const int bn = p.bn;         // columns of a tile
    const bool wide = bn > 64;   // activation stages of 64 values of K instead of 128 (shared memory)
    const uint32_t half_bytes = (uint32_t)bn * 128u, stage_bytes = wide ? half_bytes : 2u * half_bytes;  // 64 values: a 128-byte row
    const uint32_t ring_addr = tile_base + S * stage_bytes;
    uint8_t *ring = smem_raw + (ring_addr - raw_addr);
    const uint32_t R = 1u << p.raw_shift;
    const uint32_t full = bar_base, empty = bar_base + 64u, raw_full = bar_base + 128u, raw_empty = bar_base + 192u,
                   d_full = bar_base + 256u, d_empty = bar_base + 264u, share_bar = bar_base + 272u, ticket_bar = bar_base + 280u,
                   b_full = bar_base + 320u, b_empty = bar_base + 352u;  // wide tiles only
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ volatile int last_s;
    __shared__ int group_tile0[TS_MAX_GROUPS + 1];  // grouped launches: first tile of every group

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = p.split;  // > 1: the CTAs of a cluster share one tile along K
    const int cta = (int)blockIdx.x, n_cta = (int)gridDim.x;
    const bool grouped = p.group_counts != nullptr;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < S; ++i) {
            tm_mbar_init(full + 8u * i, wide ? 4 : 5);  // a group's warps, and the activation tile
            tm_mbar_init(empty + 8u * i, 1);
            tm_mbar_init(b_full + 8u * i, 1);
            tm_mbar_init(b_empty + 8u * i, 1);
        }
        for (uint32_t i = 0; i < R; ++i) {
            tm_mbar_init(raw_full + 8u * i, 1);
            tm_mbar_init(raw_empty + 8u * i, 8);
        }
        tm_mbar_init(d_full, 1);
        tm_mbar_init(d_empty, TS_CONV);
        tm_mbar_init(share_bar, TS_CONV);
        tm_mbar_init(ticket_bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (grouped && warp == TS_W_WARP) {
        ts_group_table(p, bn, group_tile0, lane);
    }
    if (warp == TS_MMA_WARP)  // (all columns are taken: the permit to allocate need not be given back)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tm_smem_u32(&tmem_slot)) : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // (In shared memory, and the converted columns in quarters, for the registers: what a thread spills misses the few KB of L1 that
    // are left.  Spilled stores and loads in bytes, before and so: Q4_K 96 + 184, 36 + 56 (64 x 4096 x 14336 18.3 -> 17.8 us); Q6_K 100 + 188,
    // 36 + 60 (37 x 14336 x 4096 27.4 -> 25.7); Q8_0 104 + 232, 88 + 120.  With twice the former the large sizes were 10 to 25 % slower.)
    __shared__ TsWork work_s;
    if (threadIdx.x == 0) work_s = ts_work(p, grouped, group_tile0, bn, cta, n_cta);
    __syncthreads();
    const TsWork &work = work_s;
    const int KS = p.slabs, u0 = work.u0, u1 = work.u1;
    auto tile_of = [&](int tile) { return work.tile(p, tile); };

    bool ok = true;
    int err_code = 0;
    if (warp == TS_B_WARP) {
        // ------------------------------ activation tiles ------------------------------
        if (lane == 0) {
            // (without work too: the kernel behind relies on this grid's end to order it behind the staging kernel)
            asm volatile("griddepcontrol.wait;" ::: "memory");
            uint32_t s = 0;
            for (int u = u0; u < u1 && ok;) {
                const int tile = u / KS, k_lo = u - tile * KS, k_hi = min(KS, k_lo + (u1 - u));
                const TsTile t = tile_of(tile);
                const int per = wide ? 4 : 2, step = 256 / per;
                for (int k = per * k_lo; k < per * k_hi; ++k, ++s) {
                    const uint32_t st = s & (S - 1), use = s / S;
                    if (use >= 1 && !ts_wait((wide ? b_empty : empty) + 8u * st, (use - 1) & 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t dst = tile_base + st * stage_bytes, bar = (wide ? b_full : full) + 8u * st;
                    tm_mbar_expect_tx(bar, stage_bytes);
                    tm_tma_load_2d(dst, &maps.x, k * step, t.t_row0, bar);
                    if (!wide) tm_tma_load_2d(dst + half_bytes, &maps.x, k * step + 64, t.t_row0, bar);
                }
                u += k_hi - k_lo;
            }
            err_code = 6;
        }
        __syncwarp();
    } else if (warp == TS_W_WARP) {
        // ------------------------------ packed weight slabs ------------------------------
        ok = ts_stream_slabs<KIND>(maps, p, work, loose, ring_addr, ring, SLAB, raw_full, raw_empty, lane);
        err_code = 10;
        __syncwarp();
    } else if (warp == TS_MMA_WARP) {
        // ------------------------------ MMA issuer ------------------------------
        const uint64_t b_desc0 = tm_smem_desc(tile_base);
        const uint32_t half_step = half_bytes >> 4;
        if (tm_elect_one()) {
            uint32_t slab = 0, idesc = 0;  // slabs of this CTA's range issued so far
            // Stage slots are compile-time constants here: with ring positions computed at run time a commit costs the issuing
            // thread about 400 cycles before its next instruction, with constants about 200 (with the barrier wait); the eight
            // MMAs of a stage take 4 bn.
            auto issue = [&](auto first_slot, auto is_wide, bool start, bool stop) {
                constexpr uint32_t SLOT = decltype(first_slot)::value;
                constexpr bool WIDE = decltype(is_wide)::value;
#pragma unroll
                for (uint32_t hs = 0; hs < 2; ++hs) {
                    const uint32_t st = SLOT + hs;
                    ok = ok && ts_wait(full + 8u * st, (slab >> 1) & 1u);
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        if (WIDE) ok = ok && ts_wait(b_full + 8u * (2 * hs + h), slab & 1u);
                        if (!ok) return;
                        if (WIDE || h == 0) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint64_t b = WIDE ? b_desc0 + (2 * hs + h) * half_step : b_desc0 + (2 * st + h) * half_step;
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i)
                            ts_mma(tmem, tmem + TS_D_COLS + st * 64u + 32u * h + 8u * i, b + 2u * i, idesc,
                                   (i == 0 && h == 0 && hs == 0 && start) ? 0u : 1u);
                        if (WIDE) tm_commit(b_empty + 8u * (2 * hs + h));
                    }
                    tm_commit(empty + 8u * st);
                    if (hs == 1 && stop) tm_commit(d_full);
                }
                ++slab;
            };
            using Slot0 = std::integral_constant<uint32_t, 0>;
            using Slot2 = std::integral_constant<uint32_t, 2>;
            int seg = 0;
            for (int u = u0; u < u1 && ok; ++seg) {
                const int tile = u / KS, k_lo = u - tile * KS, n = min(KS, k_lo + (u1 - u)) - k_lo;
                const int cols = (tile_of(tile).t_count + 15) & ~15;
                idesc = (1u << 4) | ((uint32_t)(cols >> 3) << 17) | ((uint32_t)(TS_ROWS >> 4) << 24);
                if (seg >= 1) ok = ts_wait(d_empty, (uint32_t)(seg - 1) & 1u);
                for (int k = 0; k < n && ok; ++k) {
                    if (wide) {
                        if (slab & 1u) issue(Slot2(), std::true_type(), k == 0, k == n - 1);
                        else issue(Slot0(), std::true_type(), k == 0, k == n - 1);
                    } else {
                        if (slab & 1u) issue(Slot2(), std::false_type(), k == 0, k == n - 1);
                        else issue(Slot0(), std::false_type(), k == 0, k == n - 1);
                    }
                }
                u += n;
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        err_code = 7;
        __syncwarp();
    } else {
        // ------------------------------ converters and epilogue ------------------------------
        const int group = warp >> 2, q = warp & 3;
        const int r = 32 * q + lane;                              // TMEM lane of this thread
        const int fr = loose ? (r >> 4) + 8 * (r & 15) : r;       // weight row it holds, inside the CTA's tile
        const uint32_t lane_addr = tmem + ((uint32_t)(32 * q) << 16);
        uint32_t shares = 0;  // shares of cut tiles handled so far: the phase of share_bar / ticket_bar

        auto epilogue = [&](int seg, int u_lo, int u_hi) {  // units [u_lo, u_hi) of one tile
            const int tile = u_lo / KS;
            const TsTile t = tile_of(tile);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const TsJob &jb = p.jobs[t.job];
            const bool live = fr < t.rows;
            const int f = t.f0 + fr;
            const float bias = (live && jb.bias != nullptr) ? jb.bias[f] : 0.0f;
            // the scales of this warp's columns: chunk group + 4 i in lanes 16 (i % 2) .. of scale[i / 2]
            float scale[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int col = 16 * (group + 8 * i + 4 * (lane >> 4)) + (lane & 15);
                scale[i] = col < t.t_count ? p.rowscale[t.t_row0 + col] : 0.0f;
            }
            ok = ts_wait(d_full, (uint32_t)seg & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // column chunks of 16 tokens, chunk c to group c % 4, two chunks at a time (registers); the accumulator is free for
            // the next tile's MMAs once the last pair has been read
            const int chunks = (t.t_count + 15) >> 4;
            float *outp = jb.out + (size_t)t.t_row0 * jb.ldo + f;
            const bool whole = u_hi - u_lo == KS;
            // A share of a tile goes into this CTA's slot (0: the share its range starts with, 1: the one it ends with).
            auto slot = [&](int c, int which) -> float * {
                return p.partial + ((size_t)c * 2 + which) * ((size_t)TS_ROWS * bn);
            };
            float *mine = split > 1 ? nullptr : slot(cta, u_lo == u0 ? 0 : 1) + r;
            // (split tiles: the activation ring is idle by now and holds the share for the other CTAs of the cluster)
            float *shared_share = (float *)(smem_raw + (tile_base - raw_addr)) + r;
#pragma unroll 1
            for (int cb = group; ; cb += 8) {
                const float sc = cb == group ? scale[0] : scale[1];
                uint32_t v[2][16];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (cb + 4 * i < chunks) ts_ld16(lane_addr + 16u * (uint32_t)(cb + 4 * i), v[i]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (cb + 8 >= chunks) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tm_mbar_arrive(d_empty);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int c = cb + 4 * i;
                    if (c >= chunks) continue;
                    if (whole) {
                        ts_store16(outp, jb.ldo, 16 * c, t.t_count, live, bias, sc, 16 * i, v[i]);
                    } else if (split > 1) {
#pragma unroll
                        for (int jj = 0; jj < 16; ++jj) shared_share[(16 * c + jj) * TS_ROWS] = __uint_as_float(v[i][jj]);
                    } else {
#pragma unroll
                        for (int jj = 0; jj < 16; ++jj) __stcg(mine + (16 * c + jj) * TS_ROWS, __uint_as_float(v[i][jj]));
                    }
                }
                if (cb + 8 >= chunks) break;
            }
            if (whole || split > 1) return;
            // Then a ticket; the CTA that draws the last one of the tile adds the shares in the order of K.
            // (mbarriers instead of a named barrier: a warp that gave up must not leave the others waiting for good)
            __threadfence();
            __syncwarp();
            if (lane == 0) tm_mbar_arrive(share_bar);
            const TsOwners own = ts_owners(work, tile, KS);
            if (warp == 0) {
                ok = ts_wait(share_bar, shares & 1u);
                ok = __all_sync(0xffffffffu, ok);
            }
            if (threadIdx.x == 0 && ok) {
                int *ctr = p.counters + own.first;
                const int ticket = atomicAdd(ctr, 1);
                last_s = ticket == own.last - own.first;
                if (last_s) *ctr = 0;  // ready for the next launch
                tm_mbar_arrive(ticket_bar);
            }
            __syncwarp();
            if (ok) ok = ts_wait(ticket_bar, shares & 1u);
            ok = __all_sync(0xffffffffu, ok);
            ++shares;
            if (!ok || !last_s) return;
            __threadfence();
#pragma unroll 1
            for (int c = group; c < chunks; c += 4) {
                float acc[16];
#pragma unroll
                for (int jj = 0; jj < 16; ++jj) acc[jj] = 0.0f;
#pragma unroll 2
                for (int k = own.first; k <= own.last; ++k) {
                    // a CTA whose range starts inside the tile, or exactly at its start, holds the share in slot 0
                    const float *from = slot(k, ts_share_slot(work, tile, KS, k)) + (16 * c) * TS_ROWS + r;
                    float w[16];
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) w[jj] = __ldcg(from + jj * TS_ROWS);
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) acc[jj] += w[jj];
                }
                uint32_t v[16];
#pragma unroll
                for (int jj = 0; jj < 16; ++jj) v[jj] = __float_as_uint(acc[jj]);
                const int i = (c - group) >> 2;
                ts_store16(outp, jb.ldo, 16 * c, t.t_count, live, bias, i < 2 ? scale[0] : scale[1], 16 * (i & 1), v);
            }
        };

        // Slabs group >> 1, + 2, ... of the CTA's range.  A group converts its next slab before it turns to the epilogue of a
        // finished segment (the part of one tile in the range), so that the MMAs find the ring filled when the accumulator
        // is free again.  The last round converts nothing and runs the epilogues that are left.
        const int half = group & 1, n_slabs = u1 - u0;
        int pend_seg = 0, pend_u = u0;  // first segment whose epilogue is outstanding
        int tile = u0 / KS, seg = 0;    // of slab j
        uint32_t row_at = 0, row_phase = 0, row_mask = 15u;  // this thread's row in a slab, and the offset of its first slab's data there
        auto find_row = [&](int tl) {
            const TsTile t = tile_of(tl);
            const TsJob &jb = p.jobs[t.job];
            const int rest0 = jb.F & ~7, f = t.f0 + fr;
            const uintptr_t at = (uintptr_t)jb.w + (size_t)(t.w_row0 + fr) * p.row_bytes;
            const bool rest = f >= rest0 && f < jb.F;  // (see the slab producer)
            row_at = (uint32_t)(rest ? TS_ROWS + f - rest0 : r) * SL::LOOSE_PITCH;
            row_mask = rest ? 3u : 15u;
            row_phase = (uint32_t)at & row_mask;
        };
        row_at = (uint32_t)r * SL::PITCH;
        if (loose && n_slabs > 0) find_row(tile);
#pragma unroll 1
        for (int j = group >> 1; ok; j += 2) {
            const bool tail = j >= n_slabs;
            if (!tail) {
                if (u0 + j >= (tile + 1) * KS) {
                    const int to = (u0 + j) / KS;
                    seg += to - tile;
                    tile = to;
                    if (loose) find_row(tile);
                }
                const uint32_t rs = (uint32_t)j & (R - 1u);
                ok = ts_wait(raw_full + 8u * rs, ((uint32_t)j >> p.raw_shift) & 1u);
                const uint8_t *rowp = ring + rs * SLAB + row_at;
                auto done = [&] {
                    __syncwarp();
                    if (lane == 0) tm_mbar_arrive(raw_empty + 8u * rs);
                };
                auto emit = [&](int t, const uint32_t (&o)[16]) {
                    if (t == 0) {
                        // The slot's previous MMAs: waited for only now, the conversion has hidden some of it.
                        if (ok && j >= 2) ok = ts_wait(empty + 8u * group, ((uint32_t)(j >> 1) - 1u) & 1u);
                        ok = __all_sync(0xffffffffu, ok);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    if (ok) ts_st16(lane_addr + TS_D_COLS + (uint32_t)group * 64u + 16u * (uint32_t)t, o);
                };
                if constexpr (KIND == KIND_Q4_K) {
                    ts_conv_q4k(rowp, half, done, emit);
                } else if constexpr (KIND == KIND_Q6_K) {
                    const int k = u0 + j - tile * KS;
                    const uint32_t phase = (row_phase + (uint32_t)(k * SL::BYTES)) & row_mask;
                    ts_conv_q6k<loose>(rowp + phase, phase, half, done, emit);
                } else {
                    const int n_blk = p.nb - 8 * (u0 + j - tile * KS);
                    if (loose) ts_conv_q8_0_loose(rowp + row_phase, half, n_blk, done, emit);
                    else if (half == 0) ts_conv_q8_0<0>(rowp, n_blk, done, emit);
                    else ts_conv_q8_0<1>(rowp, n_blk, done, emit);
                }
                if (!ok) break;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tm_mbar_arrive(full + 8u * group);
            }
#pragma unroll 1
            while (ok && pend_u < u1 && (tail || pend_seg < seg)) {
                const int e = min((pend_u / KS + 1) * KS, u1);
                epilogue(pend_seg, pend_u, e);
                pend_u = e;
                ++pend_seg;
            }
            if (tail) break;
        }
        err_code = 8;
    }
    if (!ok) {
        if (lane == 0) atomicExch(p.err, err_code);
        abort_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (abort_flag) {
        // A wait ran out and some agent stopped early: bulk copies may still be landing in this CTA's shared memory.  Give
        // them time to finish before the CTA (and its shared memory) goes away.
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (split > 1) {
        __syncwarp();
        ts_cluster_sync();  // the shares of the split tile are complete
        // Every CTA of the cluster adds the shares of its part of the tile's columns, in the order of K, out of the shared memories.
        const TsTile t = tile_of(cta / split);
        const TsJob &jb = p.jobs[t.job];
        const int part = cta - cta / split * split, c_lo = t.t_count * part / split, c_hi = t.t_count * (part + 1) / split;
        const int r = threadIdx.x & (TS_ROWS - 1), fr = loose ? (r >> 4) + 8 * (r & 15) : r, f = t.f0 + fr;
        if (threadIdx.x < 512 && fr < t.rows) {
            uint32_t from[TS_MAX_SPLIT];
#pragma unroll
            for (int i = 0; i < TS_MAX_SPLIT; ++i)
                from[i] = i < split ? ts_mapa(tile_base + 4u * (uint32_t)r, (uint32_t)i) : 0u;
            const float bias = jb.bias != nullptr ? jb.bias[f] : 0.0f;
            int c = c_lo + (int)(threadIdx.x >> 7);
            if (split == 2) {
                // Pairs share wide tiles: eight columns at a time, so that sixteen loads are under way (500 x 4096 x 4096 Q4_K, 125
                // columns for each CTA: 31.1 -> 27.6 us; with four and eight CTAs to a tile it was slower, 13.4 -> 13.7 at 64 tokens).
                constexpr int BATCH = 8;
                for (; c < c_hi; c += 4 * BATCH) {
                    float v[2][BATCH];
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int j = 0; j < BATCH; ++j) {
                            v[i][j] = 0.0f;
                            if (c + 4 * j < c_hi)
                                asm volatile("ld.shared::cluster.f32 %0, [%1];"
                                             : "=f"(v[i][j]) : "r"(from[i] + (uint32_t)(c + 4 * j) * (TS_ROWS * 4u)) : "memory");
                        }
#pragma unroll
                    for (int j = 0; j < BATCH; ++j)
                        if (c + 4 * j < c_hi)
                            jb.out[(size_t)(t.t_row0 + c + 4 * j) * jb.ldo + f] = (v[0][j] + v[1][j]) * p.rowscale[t.t_row0 + c + 4 * j] + bias;
                }
            }
            for (; c < c_hi; c += 4) {
                float v[TS_MAX_SPLIT];
#pragma unroll
                for (int i = 0; i < TS_MAX_SPLIT; ++i) {
                    v[i] = 0.0f;
                    if (i < split)
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[i]) : "r"(from[i] + (uint32_t)c * (TS_ROWS * 4u)) : "memory");
                }
                float acc = v[0];
#pragma unroll
                for (int i = 1; i < TS_MAX_SPLIT; ++i)
                    if (i < split) acc += v[i];
                jb.out[(size_t)(t.t_row0 + c) * jb.ldo + f] = acc * p.rowscale[t.t_row0 + c] + bias;
            }
        }
        __syncwarp();
        ts_cluster_sync();  // nobody leaves while its share is being read
    }
    if (warp == TS_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
size_t gemm_ts_workspace_bytes() {
    // two shares of 128 x 256 floats per CTA, and a ticket each
    return (size_t)device_sm_count() * 2 * TS_ROWS * 256 * sizeof(float);
}

bool gemm_ts_supported(int kind, const void *W, int T, int K, int F) {
    if (!kind_supported(kind) || T < 1 || K < 1 || F < 1 || encode_tiled_fn() == nullptr) return false;
    const long rb = (long)((K + block_values(kind) - 1) / block_values(kind)) * block_bytes(kind);
    return kind != KIND_Q4_K || (((uintptr_t)W & 15) == 0 && rb % 16 == 0);
}

bool ts_loose(int kind, const void *W, long row_bytes) {
    return kind != KIND_Q4_K && (((uintptr_t)W & 15) != 0 || row_bytes % 16 != 0);
}

template <int KIND, bool LOOSE>
static cudaError_t ts_launch(const TsMaps &maps, TsParams &p, int n_cta, int dev, cudaStream_t s) {
    const int stage_bytes = (p.bn > 64 ? 1 : 2) * p.bn * 128;
    const int fixed = 16 + 512 + 1024 + TS_STAGES * stage_bytes;
    constexpr int slab = ts_slab_bytes<KIND>(LOOSE);
    constexpr int MOST = 224 * 1024;
    p.raw_shift = fixed + 4 * slab <= MOST ? 2 : 1;
    const int smem = fixed + (slab << p.raw_shift);
    static std::atomic<uint64_t> configured{0};  // devices on which the kernel may use that much shared memory
    const bool known = dev >= 0 && dev < 64;
    if (!known || !(configured.load(std::memory_order_relaxed) >> dev & 1)) {
        if (cudaError_t e = cudaFuncSetAttribute(gemm_ts_kernel<KIND, LOOSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST)) return e;
        if (known) configured.fetch_or((uint64_t)1 << dev, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_cta, 1, 1);
    cfg.blockDim = dim3(TS_THREADS, 1, 1);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.split > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_ts_kernel<KIND, LOOSE>, maps, p);
}

static cudaError_t ts_dispatch(int kind, const TsMaps &maps, TsParams &p, int n_cta, int dev, cudaStream_t s) {
    switch (kind) {
    case KIND_Q4_K: return ts_launch<KIND_Q4_K, false>(maps, p, n_cta, dev, s);
    case KIND_Q6_K: return p.loose ? ts_launch<KIND_Q6_K, true>(maps, p, n_cta, dev, s) : ts_launch<KIND_Q6_K, false>(maps, p, n_cta, dev, s);
    default: return p.loose ? ts_launch<KIND_Q8_0, true>(maps, p, n_cta, dev, s) : ts_launch<KIND_Q8_0, false>(maps, p, n_cta, dev, s);
    }
}

cudaError_t ts_encode(CUtensorMap *m, CUtensorMapDataType type, const void *base, cuuint64_t d0, cuuint64_t d1,
                             cuuint64_t stride, cuuint32_t b0, cuuint32_t b1, CUtensorMapSwizzle sw) {
    const cuuint64_t dims[2] = {d0, d1}, strides[1] = {stride};
    const cuuint32_t box[2] = {b0, b1}, es[2] = {1, 1};
    return encode_tiled_fn()(m, type, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
        ? cudaSuccess
        : cudaErrorInvalidValue;
}

// Tensor map of a weight matrix: [rows][row bytes], or, for rows that are not 16-byte multiples, [rows / 8][eight rows].
cudaError_t ts_encode_weights(int kind, CUtensorMap *m, const void *W, long row_bytes, size_t rows, bool loose) {
    const int unit = kind == KIND_Q8_0 ? 4 : 1;  // a box is at most 256 elements wide
    const CUtensorMapDataType type = kind == KIND_Q8_0 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    if (!loose) {
        const int pitch = kind == KIND_Q4_K ? TsSlab<KIND_Q4_K>::PITCH : kind == KIND_Q6_K ? TsSlab<KIND_Q6_K>::PITCH : TsSlab<KIND_Q8_0>::PITCH;
        return ts_encode(m, type, W, (cuuint64_t)(row_bytes / unit), rows, (cuuint64_t)row_bytes, (cuuint32_t)(pitch / unit), TS_ROWS,
                         CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    const int pitch = kind == KIND_Q6_K ? TsSlab<KIND_Q6_K>::LOOSE_PITCH : TsSlab<KIND_Q8_0>::LOOSE_PITCH;
    const long shift = (long)((uintptr_t)W & 15), wide = shift + 8 * row_bytes;
    // (fewer than eight rows: all of them are fetched with plain loads; the map only has to be valid, and out of range)
    const size_t eights = rows / 8;
    return ts_encode(m, type, (const void *)((uintptr_t)W & ~(uintptr_t)15), (cuuint64_t)(eights > 0 ? (wide + unit - 1) / unit : 16 / unit),
                     eights > 0 ? eights : 1, (cuuint64_t)(8 * row_bytes), (cuuint32_t)(pitch / unit), TS_ROWS / 8, CU_TENSOR_MAP_SWIZZLE_NONE);
}

cudaError_t launch_gemm_ts(int kind, const GemvJobSpec *jobs, int n_jobs, const __half *xh, const float *rowscale, int ldxh,
                           int T, int K, float *partial, int *counters, int *err_flag, cudaStream_t s) {
    if (n_jobs < 1 || n_jobs > TS_MAX_JOBS) return cudaErrorInvalidValue;
    TsParams p;
    TsMaps maps;
    memset(&p, 0, sizeof(p));
    int F[TS_MAX_JOBS];
    for (int j = 0; j < n_jobs; ++j) F[j] = jobs[j].F;
    int dev;
    const TsPlan pl = ts_plan(kind, T, K, F, n_jobs, device_sm_count(&dev));
    if ((long)(pl.t_tiles - 1) * pl.bn >= T) return cudaErrorInvalidValue;  // a tile without tokens is no MMA
    p.nb = (K + block_values(kind) - 1) / block_values(kind);
    p.row_bytes = (long)p.nb * block_bytes(kind);
    p.slabs = (p.nb * block_values(kind) + TS_SLAB_K - 1) / TS_SLAB_K;
    p.rowscale = rowscale;
    p.partial = partial;
    p.counters = counters;
    p.err = err_flag;
    p.n_jobs = n_jobs;
    p.T = T;
    p.bn = pl.bn;
    p.t_tiles = pl.t_tiles;
    p.split = pl.split;
    p.whole = pl.whole;
    for (int j = 0; j < n_jobs; ++j) p.loose |= ts_loose(kind, jobs[j].W, p.row_bytes);
    int row_tiles = 0;
    for (int j = 0; j < n_jobs; ++j) {
        p.jobs[j] = TsJob{(const uint8_t *)jobs[j].W, jobs[j].out, jobs[j].bias, jobs[j].F, jobs[j].ldo, row_tiles};
        row_tiles += (jobs[j].F + TS_ROWS - 1) / TS_ROWS;
        if (cudaError_t e = ts_encode_weights(kind, &maps.w[j], jobs[j].W, p.row_bytes, (size_t)jobs[j].F, p.loose != 0)) return e;
    }
    p.tiles = row_tiles * pl.t_tiles;
    if (cudaError_t e = ts_encode(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, xh, ldxh, T, (cuuint64_t)ldxh * 2, 64, pl.bn,
                                  CU_TENSOR_MAP_SWIZZLE_128B))
        return e;
    return ts_dispatch(kind, maps, p, pl.n_cta, dev, s);
}

bool gemm_ts_grouped_supported(int kind, const void *W, int K, int F) {
    if (!gemm_ts_supported(kind, W, 1, K, F)) return false;
    return F % 8 == 0 || !ts_loose(kind, W, (long)((K + block_values(kind) - 1) / block_values(kind)) * block_bytes(kind));
}

// What grouped launches share: the weights and the tiles (activations and their map are the caller's).
cudaError_t ts_grouped_params(int kind, const GemvJobSpec *jobs, int n_jobs, int n_groups, int total_rows, int K,
                              const int *group_counts, const int *group_offsets, TsParams &p, TsMaps &maps) {
    memset(&p, 0, sizeof(p));
    p.nb = (K + block_values(kind) - 1) / block_values(kind);
    p.row_bytes = (long)p.nb * block_bytes(kind);
    p.slabs = (p.nb * block_values(kind) + TS_SLAB_K - 1) / TS_SLAB_K;
    p.n_jobs = n_jobs;
    p.split = 1;
    p.T = total_rows;
    p.groups = n_groups;
    p.group_counts = group_counts;
    p.group_offsets = group_offsets;
    for (int j = 0; j < n_jobs; ++j) {
        p.loose |= ts_loose(kind, jobs[j].W, p.row_bytes);
        if (!gemm_ts_grouped_supported(kind, jobs[j].W, K, jobs[j].F)) return cudaErrorNotSupported;
    }
    if (p.loose)
        for (int j = 0; j < n_jobs; ++j)
            if (jobs[j].F % 8 != 0) return cudaErrorNotSupported;
    for (int j = 0; j < n_jobs; ++j) {
        p.jobs[j] = TsJob{(const uint8_t *)jobs[j].W, jobs[j].out, jobs[j].bias, jobs[j].F, jobs[j].ldo, p.row_tiles};
        p.row_tiles += (jobs[j].F + TS_ROWS - 1) / TS_ROWS;
        if (cudaError_t e = ts_encode_weights(kind, &maps.w[j], jobs[j].W, p.row_bytes, (size_t)jobs[j].F * n_groups, p.loose != 0))
            return e;
    }
    return cudaSuccess;
}

// n_groups matmuls over stacked weight matrices (MoE experts): group g multiplies its group_counts[g] rows of xh (from row
// group_offsets[g], both device data) with the weight rows [g * F, (g + 1) * F) of every job.
cudaError_t launch_gemm_ts_grouped(int kind, const GemvJobSpec *jobs, int n_jobs, int n_groups, const __half *xh, const float *rowscale,
                                   int ldxh, int total_rows, int K, const int *group_counts, const int *group_offsets,
                                   float *partial, int *counters, int *err_flag, cudaStream_t s) {
    if (n_groups <= 0 || total_rows <= 0) return cudaSuccess;
    if (n_jobs < 1 || n_jobs > TS_MAX_JOBS) return cudaErrorInvalidValue;
    if (n_groups > TS_MAX_GROUPS) {  // the kernel keeps a table of the groups' tiles
        for (int g = 0; g < n_groups; g += TS_MAX_GROUPS) {
            const int n = n_groups - g < TS_MAX_GROUPS ? n_groups - g : TS_MAX_GROUPS;
            GemvJobSpec part[TS_MAX_JOBS];
            for (int j = 0; j < n_jobs; ++j) {
                part[j] = jobs[j];
                part[j].W = (const uint8_t *)jobs[j].W +
                    (size_t)g * jobs[j].F * ((K + block_values(kind) - 1) / block_values(kind)) * block_bytes(kind);
            }
            if (cudaError_t e = launch_gemm_ts_grouped(kind, part, n_jobs, n, xh, rowscale, ldxh, total_rows, K, group_counts + g,
                                                       group_offsets + g, partial, counters, err_flag, s))
                return e;
        }
        return cudaSuccess;
    }
    TsParams p;
    TsMaps maps;
    if (cudaError_t e = ts_grouped_params(kind, jobs, n_jobs, n_groups, total_rows, K, group_counts, group_offsets, p, maps))
        return e;
    // The counts are not known here: tiles for an even spread, up to 256 tokens.
    const int even = (total_rows + n_groups - 1) / n_groups;
    p.bn = even > 96 ? 256 : even > 48 ? 128 : 64;
    p.rowscale = rowscale;
    p.partial = partial;
    p.counters = counters;
    p.err = err_flag;
    if (cudaError_t e = ts_encode(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, xh, ldxh, total_rows, (cuuint64_t)ldxh * 2, 64,
                                  p.bn, CU_TENSOR_MAP_SWIZZLE_128B))
        return e;
    int dev;
    const int sms = device_sm_count(&dev);
    return ts_dispatch(kind, maps, p, sms, dev, s);
}

}  // namespace mcu

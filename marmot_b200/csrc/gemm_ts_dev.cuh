// What the tcgen05 matmuls with weights in tensor memory (gemm_ts.cu: fp16, gemm_ti.cu: integers) have in common: the packed
// weight slabs in shared memory, the division of the work, tensor-memory loads and stores.
#pragma once

#include "common.cuh"
#include "gemm_ts.h"
#include "tma_utils.cuh"

namespace mcu {

// A slab in shared memory: BYTES of every row, BOX bytes fetched (a 16-byte aligned window that covers them) and the pitch.  The
// pitch is an odd number of 16-byte units, so that 16-byte loads of a warp's 32 rows are conflict free.
template <int KIND>
struct TsSlab;
template <>
struct TsSlab<KIND_Q4_K> {
    static constexpr int BYTES = 144, PITCH = 144, LOOSE_PITCH = 144;
};
template <>
struct TsSlab<KIND_Q6_K> {
    static constexpr int BYTES = 210, PITCH = 240, LOOSE_PITCH = 240;
};
template <>
struct TsSlab<KIND_Q8_0> {
    static constexpr int BYTES = 272, PITCH = 272, LOOSE_PITCH = 304;  // loose: rows that start anywhere
};
template <int KIND>
constexpr int ts_slab_bytes(bool loose) {  // loose slabs keep the up to seven last rows of the matrix behind the 128
    return ((loose ? (TS_ROWS + 8) * TsSlab<KIND>::LOOSE_PITCH : TS_ROWS * TsSlab<KIND>::PITCH) + 16 + 127) / 128 * 128;
}

// N words from byte `phase` (even, below 16, the same in all threads) behind a 16-byte boundary.  With the rows' pitch, 16-byte loads are
// conflict free, where words read one by one lie four to a bank: 120 wavefronts for a warp's half of a Q6_K slab, 48 so (37 x 14336 x 4096
// 29.3 -> 27.4 us, 8 x 4096 x 14336 23.7 -> 21.0).
template <int N, int WO>
__device__ __forceinline__ void ts_shift_words(const uint32_t *w, uint32_t sh, uint32_t (&out)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = __funnelshift_r(w[WO + i], w[WO + i + 1], sh);
}
template <int N>
__device__ __forceinline__ void ts_lds_phase(const uint8_t *p, uint32_t phase, uint32_t (&out)[N]) {
    constexpr int CHUNKS = (N + 4) / 4;  // words phase / 4 .. phase / 4 + N
    uint32_t w[4 * CHUNKS];
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
        const uint4 v = *(const uint4 *)(p + 16 * i);
        w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
    }
    const uint32_t sh = (phase & 2u) * 8u;
    switch (phase >> 2) {
    case 0: ts_shift_words<N, 0>(w, sh, out); break;
    case 1: ts_shift_words<N, 1>(w, sh, out); break;
    case 2: ts_shift_words<N, 2>(w, sh, out); break;
    default: ts_shift_words<N, 3>(w, sh, out); break;
    }
}

// ---- PTX wrappers ----
__device__ __forceinline__ void ts_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t ts_mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Bounded wait.
__device__ __forceinline__ bool ts_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < 1u << 17; ++i) {  // a try suspends the thread for up to 20 us
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void ts_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
        "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void ts_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void ts_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

// The first tile of every group of a grouped launch (one warp).  May be called before griddepcontrol.wait: the staging kernel ahead lets this one start only after its own wait, when the
// kernels that wrote the counts are complete (stage_begin in act_quant.cu).
__device__ __forceinline__ void ts_group_table(const TsParams &p, int bn, int *group_tile0, int lane) {
    int base = 0;
    for (int g0 = 0; g0 < p.groups; g0 += 32) {
        const int g = g0 + lane;
        int n = g < p.groups ? (p.group_counts[g] + bn - 1) / bn * p.row_tiles : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, n, o);
            if (lane >= o) n += up;
        }
        if (g < p.groups) group_tile0[g + 1] = base + n;
        base += __shfl_sync(0xffffffffu, n, 31);
    }
    if (lane == 0) group_tile0[0] = 0;
}

// The slab producer (one warp): every slab of the CTA's range, in order, into the ring.
template <int KIND>
__device__ __forceinline__ bool ts_stream_slabs(const TsMaps &maps, const TsParams &p, const TsWork &work, bool loose, uint32_t ring_addr,
                                                uint8_t *ring, uint32_t SLAB, uint32_t raw_full, uint32_t raw_empty, int lane) {
    using SL = TsSlab<KIND>;
    const int KS = p.slabs, u0 = work.u0, u1 = work.u1;
    const uint32_t R = 1u << p.raw_shift;
    bool ok = true;
    uint32_t j = 0;
    for (int u = u0; u < u1 && ok;) {
        const int tile = u / KS, k_lo = u - tile * KS, k_hi = min(KS, k_lo + (u1 - u));
        const TsTile t = work.tile(p, tile);
        const TsJob &jb = p.jobs[t.job];
        const int rest0 = jb.F & ~7;  // loose rows: the last ones, not a whole group of eight, are fetched with plain loads
        const int rest_lo = max(t.f0, rest0), rest_hi = loose ? min(jb.F, t.f0 + TS_ROWS) : rest_lo;
        for (int k = k_lo; k < k_hi; ++k, ++j) {
            const uint32_t rs = j & (R - 1u), use = j >> p.raw_shift;
            if (use >= 1) ok = ts_wait(raw_empty + 8u * rs, (use - 1) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t dst = ring_addr + rs * SLAB, bar = raw_full + 8u * rs;
            for (int f = rest_lo; f < rest_hi; ++f) {
                const uintptr_t row = (uintptr_t)jb.w + (size_t)f * p.row_bytes + (size_t)k * SL::BYTES;
                const int bytes = min(SL::BYTES, (int)(p.row_bytes - (long)k * SL::BYTES)) + (int)(row & 3u);
                uint8_t *to = ring + (size_t)rs * SLAB + (size_t)(TS_ROWS + f - rest0) * SL::LOOSE_PITCH;
                for (int w = lane; 4 * w < bytes; w += 32) *(uint32_t *)(to + 4 * w) = *(const uint32_t *)((row & ~(uintptr_t)3) + 4 * w);
            }
            __syncwarp();
            if (lane == 0) {
                if (!loose) {
                    tm_mbar_expect_tx(bar, (uint32_t)(TS_ROWS * SL::PITCH));
                    const int x = KIND == KIND_Q8_0 ? k * (SL::BYTES / 4) : (k * SL::BYTES) & ~15;
                    tm_tma_load_2d(dst, &maps.w[t.job], x, t.w_row0, bar);
                } else {
                    tm_mbar_expect_tx(bar, (uint32_t)(TS_ROWS * SL::LOOSE_PITCH));
                    const uint32_t shift = (uint32_t)((uintptr_t)jb.w & 15u);
                    for (int e = 0; e < 8; ++e) {
                        const long at = (long)shift + (long)e * p.row_bytes + (long)k * SL::BYTES;
                        const int x = (int)(at & ~15l) / (KIND == KIND_Q8_0 ? 4 : 1);
                        tm_tma_load_2d(dst + (uint32_t)(e * (TS_ROWS / 8) * SL::LOOSE_PITCH), &maps.w[t.job], x, t.w_row0 >> 3, bar);
                    }
                }
            }
        }
        u += k_hi - k_lo;
    }
    return ok;
}

}  // namespace mcu

// Quantized matmul for a handful of tokens on the integer tensor core (tcgen05.mma kind::i8), Q4_K and Q6_K weights in tensor
// memory: every 32-value (Q4_K) or 16-value (Q6_K) sub-block dot product is an exact 32-bit integer, as in the reference's
// vec_dot_q4_k_q8_k / vec_dot_q6_k_q8_k (vec_dot_impl.h:688-732,783-828); only the order of the per-block f32 terms differs.
//
// What bounds it is the weight stream.  Packed words become 8-bit operands with a mask and a shift (no conversion to fp16), and
// the tensor core leaves one 32-bit sum per weight row, token and sub-block in tensor memory; scaling those by the 6-bit (8-bit)
// sub-block scales is one multiply-add each, where the dp4a kernel needs eight dots and the mma.sync kernel a fragment shuffle.
// The Q4_K mins (sum_j m_j * bsum_j) and the offset 32 of the Q6_K quants (32 * sum_j sc_j * bsum_j) are two more MMAs: the
// sub-block sums of the activations come split as 64 * hi + lo into 8-bit values.
//
//   warps 0..7    converters, two groups of four warps; group c takes the slabs (128 rows x 256 values) j with j % 2 == c
//   warps 8..15   scalers, two groups; a unit (Q4_K: a slab, Q6_K: half a slab) to group unit % 2.  They read the integer sums,
//                 keep the f32 sums of sixteen tokens in registers and write the result.
//   warp 16       issues the MMAs: ten (Q4_K) or twelve (Q6_K) per slab of 128 rows x 32 values x 16 or 32 columns
//   warp 17       activation tiles by TMA;  warp 18  packed weight slabs by TMA (as in gemm_ts.cu)
//
// Work is divided as in gemm_ts.cu: whole tiles, a tile over a cluster, or equal ranges of slabs.
//
// Measured, staging included, against the kernels that had these calls (mma.sync, dp4a): Q4_K 8 x 4096 x 14336 19.9 -> 13.0 us
// (2.5 TB/s), 8 x 4096 x 28672 22.3 (3.0 TB/s), 16 x 4096 x 14336 22.4 -> 14.5; Q6_K 8 x 4096 x 14336 25.2 -> 18.5.  The mma.sync kernel keeps the
// calls of up to 16 tokens for which it is the faster one (gemm_i8.cu; i8_pays in gemm_plan.h).  A slab costs the Q4_K scalers and
// converters 500 to 700 cycles by their own stamps (740 by the time of a CTA with sixteen), the Q6_K ones (eighteen products of 32 columns, 4 KB of sums per row) 900 to 1800; a
// CTA's time grows by 900 and 2100 with each (ti_plan).  Those bound Q6_K, the kernel's prologue, staging launch and first loads (about
// 5 us) the small sizes.
#include "gemm_ts_dev.cuh"

#include <atomic>
#include <cstring>
#include <type_traits>

namespace mcu {

constexpr int TI_CONV = 8, TI_SCALE = 8;
constexpr int TI_MMA_WARP = TI_CONV + TI_SCALE, TI_B_WARP = TI_MMA_WARP + 1, TI_W_WARP = TI_MMA_WARP + 2;
constexpr int TI_THREADS = (TI_W_WARP + 1) * 32;
constexpr int TI_D_COLS = 160;              // a unit's integer sums: eight (four) tiles of 16 (32) columns, two of corrections
constexpr int TI_A_COLS = 80, TI_A0 = 320;  // a slab's operands: 64 columns of quants, 16 of mins / scales
constexpr int TI_B_SLOTS = 4;
template <int KIND>
constexpr uint32_t ti_b_bytes() { return KIND == KIND_Q4_K ? 6144u : 10240u; }  // [16 tokens x 128 B] boxes

__device__ __forceinline__ void ti_mma(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 0, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc) : "memory");
}
// D 32-bit integers, A and B signed bytes, M = 128
__host__ __device__ constexpr uint32_t ti_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TS_ROWS >> 4) << 24);
}
__device__ __forceinline__ void ti_ld8(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void ti_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The operands of one weight row in a slab: 64 words of quants in the order of K, then the corrections' words.
// Q4_K: sub-block 2 g in the low, 2 g + 1 in the high nibbles of bytes 32 g .. 32 g + 31.
template <class Done, class Emit>
__device__ __forceinline__ void ti_conv_q4k(const uint8_t *rowp, Done done, Emit emit) {
    const uint4 hdr = *(const uint4 *)rowp;
    uint4 q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = *(const uint4 *)(rowp + 16 + 16 * i);
    done();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t o[32];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint4 a = q[4 * h + 2 * g], b = q[4 * h + 2 * g + 1];
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                o[16 * g + i] = w[i] & 0x0F0F0F0Fu;
                o[16 * g + 8 + i] = (w[i] >> 4) & 0x0F0F0F0Fu;
            }
        }
        emit(h, o);
    }
    uint32_t c[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) c[i] = 0u;
    c[0] = hdr.z & 0x3F3F3F3Fu;  // mins 0..3, 4..7
    c[1] = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
    emit.corrections(c);
}
// Q6_K: value 128 n + 32 c + l has its low four bits in byte 64 n + 32 (c & 1) + l of ql (high nibble for c >= 2), its high two
// in bits 2 c of byte 32 n + l of qh.  The quants stay 0..63 here.
// EVEN: all rows start at byte `phase` behind a 16-byte boundary.
template <bool EVEN, class Done, class Emit>
__device__ __forceinline__ void ti_conv_q6k(const uint8_t *blk, uint32_t phase, Done done, Emit emit) {
    uint32_t sc[4];
    tm_lds_words<4>(blk + 192, sc);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        uint32_t ql[16], qh[8], o[32];
        if (EVEN) {
            ts_lds_phase<16>(blk - phase + 64 * n, phase, ql);
            ts_lds_phase<8>(blk - phase + 128 + 32 * n, phase, qh);
        } else {
            tm_lds_words<16>(blk + 64 * n, ql);
            tm_lds_words<8>(blk + 128 + 32 * n, qh);
        }
        if (n == 1) done();
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t hi = c >= 2 ? qh[j] >> (2 * c - 4) : qh[j] << (4 - 2 * c);
                o[8 * c + j] = ((ql[8 * (c & 1) + j] >> (4 * (c >> 1))) & 0x0F0F0F0Fu) | (hi & 0x30303030u);
            }
        emit(n, o);
    }
    // sixteen scales; the first eight for the first half's correction, the others for the second's
    uint32_t c[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) c[i] = 0u;
    c[0] = sc[0], c[1] = sc[1], c[8 + 2] = sc[2], c[8 + 3] = sc[3];
    emit.corrections(c);
}

// LOOSE: Q6_K rows that are not 16-byte multiples (as a branch beside the 16-byte loads of the others it cost them about 1 %: 7 x 4608 x 2176
// 12.27 us, 12.17 so).
template <int KIND, bool LOOSE>
__global__ void __launch_bounds__(TI_THREADS, 1)
gemm_ti_kernel(const __grid_constant__ TsMaps maps, const __grid_constant__ TsParams p) {
    extern __shared__ uint8_t smem_raw[];
    using SL = TsSlab<KIND>;
    constexpr bool Q4 = KIND == KIND_Q4_K;
    constexpr uint32_t B_BYTES = ti_b_bytes<KIND>();
    constexpr bool loose = LOOSE;
    const uint32_t SLAB = loose ? ts_slab_bytes<KIND>(true) : ts_slab_bytes<KIND>(false);
    const uint32_t raw_addr = tm_smem_u32(smem_raw);
    const uint32_t bar_base = (raw_addr + 15u) & ~15u;
    const uint32_t tile_base = (bar_base + 512u + 1023u) & ~1023u;
    float *sums = (float *)(smem_raw + (tile_base + TI_B_SLOTS * B_BYTES - raw_addr));  // [16][128]: group 1's part of a tile
    const uint32_t share_addr = tile_base + TI_B_SLOTS * B_BYTES + TI_COLS * TS_ROWS * 4u;
    float *shared_share = (float *)(smem_raw + (share_addr - raw_addr));  // [16][128]: this CTA's share of a split tile
    const uint32_t ring_addr = share_addr + TI_COLS * TS_ROWS * 4u;
    uint8_t *ring = smem_raw + (ring_addr - raw_addr);
    const uint32_t R = 1u << p.raw_shift;
    const uint32_t a_full = bar_base, b_full = bar_base + 16u, ab_empty = bar_base + 48u, d_full = bar_base + 80u, d_empty = bar_base + 96u,
                   seg_full = bar_base + 112u, seg_free = bar_base + 120u, share_bar = bar_base + 128u,
                   raw_full = bar_base + 144u, raw_empty = bar_base + 208u, dx_read = bar_base + 272u;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ int cut_tile[2];  // cut tiles that this CTA has to add up: of its range's start and end
    __shared__ int cut_first[2], cut_last[2], cut_slot[2];  // who has their shares, and which slot of the first one
    __shared__ int group_tile0[TS_MAX_GROUPS + 1];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = p.split, cta = (int)blockIdx.x, n_cta = (int)gridDim.x;
    const bool grouped = p.group_counts != nullptr;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 2; ++i) {
            tm_mbar_init(a_full + 8u * i, 4);
            tm_mbar_init(d_full + 8u * i, 1);
            tm_mbar_init(d_empty + 8u * i, 4);
        }
        for (uint32_t i = 0; i < TI_B_SLOTS; ++i) {
            tm_mbar_init(b_full + 8u * i, 1);
            tm_mbar_init(ab_empty + 8u * i, 1);
            tm_mbar_init(dx_read + 8u * i, Q4 ? 4 : 8);  // the scalers that read the block scales of a slot
        }
        for (uint32_t i = 0; i < R; ++i) {
            tm_mbar_init(raw_full + 8u * i, 1);
            tm_mbar_init(raw_empty + 8u * i, Q4 ? 8 : 12);
        }
        tm_mbar_init(seg_full, 4);
        tm_mbar_init(seg_free, 4);
        tm_mbar_init(share_bar, 4);  // the shares of the cut tiles at the range's start and end
        tm_mbar_init(share_bar + 8u, 4);
        abort_flag = 0;
        cut_tile[0] = cut_tile[1] = -1;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (grouped && warp == TI_W_WARP) ts_group_table(p, TI_COLS, group_tile0, lane);
    if (warp == TI_MMA_WARP)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tm_smem_u32(&tmem_slot)) : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const TsWork work = ts_work(p, grouped, group_tile0, TI_COLS, cta, n_cta);
    const int KS = p.slabs, u0 = work.u0, u1 = work.u1, n_slabs = u1 - u0;

    bool ok = true;
    int err_code = 0;
    if (warp == TI_B_WARP) {
        // ------------------------------ activation tiles ------------------------------
        // Who shares the cut tiles at this range's ends, for the scalers (which see it behind the barrier of the first tile).  Divisions in
        // 64 bits: here they pass while the kernel ahead is waited for.  Between a share and its ticket, and again for every share that was
        // read, they were 1 us of a launch with short ranges: MoE of 4 tokens on 8 experts of 512 x 1024 25.3 -> 23.2 us, 16 tokens on 4 of
        // 3584 x 1024 39.6 -> 36.5.  (In the scalers' own warps, whose loops they cost registers, FFN input of 8 95.4 -> 97.7.)
        if (lane < 2 && split == 1 && !p.whole && n_slabs > 0) {
            const int cut = (lane == 0 ? u0 : u1 - 1) / KS;
            const TsOwners own = ts_owners(work, cut, KS);
            cut_first[lane] = own.first;
            cut_last[lane] = own.last;
            cut_slot[lane] = ts_share_slot(work, cut, KS, own.first);
        }
        __syncwarp();
        if (lane == 0 && n_slabs > 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            uint32_t j = 0;
            for (int u = u0; u < u1 && ok;) {
                const int tile = u / KS, k_lo = u - tile * KS, k_hi = min(KS, k_lo + (u1 - u));
                const int row = work.tile(p, tile).t_row0;
                for (int k = k_lo; k < k_hi; ++k, ++j) {
                    const uint32_t st = j & (TI_B_SLOTS - 1), use = j / TI_B_SLOTS;
                    if (use >= 1 && !(ts_wait(ab_empty + 8u * st, (use - 1) & 1u) && ts_wait(dx_read + 8u * st, (use - 1) & 1u))) {
                        ok = false;
                        break;
                    }
                    const uint32_t dst = tile_base + st * B_BYTES, bar = b_full + 8u * st;
                    tm_mbar_expect_tx(bar, B_BYTES);
                    if constexpr (Q4) {
                        for (int i = 0; i < 3; ++i) tm_tma_load_2d(dst + 2048u * i, &maps.x, k * 384 + 128 * i, row, bar);
                    } else {
                        for (int i = 0; i < 2; ++i) {  // tokens with the even, then with the odd sub-blocks
                            tm_tma_load_2d(dst + 4096u * i, &maps.x, k * 384 + 128 * i, row, bar);
                            tm_tma_load_2d(dst + 4096u * i + 2048u, &maps.x, k * 384 + 128 * i, p.T + row, bar);
                        }
                        tm_tma_load_2d(dst + 8192u, &maps.x, k * 384 + 256, row, bar);
                    }
                }
                u += k_hi - k_lo;
            }
            err_code = 46;
        }
        __syncwarp();
    } else if (warp == TI_W_WARP) {
        ok = ts_stream_slabs<KIND>(maps, p, work, loose, ring_addr, ring, SLAB, raw_full, raw_empty, lane);
        err_code = 47;
        __syncwarp();
    } else if (warp == TI_MMA_WARP) {
        // ------------------------------ MMA issuer ------------------------------
        const uint64_t b_desc0 = tm_smem_desc(tile_base);
        if (tm_elect_one()) {
            auto issue = [&](auto slot, uint32_t j) {  // (slots as constants: see the issuer of gemm_ts.cu)
                constexpr uint32_t SLOT = decltype(slot)::value, A = TI_A0 + (SLOT & 1u) * TI_A_COLS;
                const uint64_t b = b_desc0 + SLOT * (B_BYTES >> 4);
                ok = ok && ts_wait(b_full + 8u * SLOT, (j >> 2) & 1u) && ts_wait(a_full + 8u * (SLOT & 1u), (j >> 1) & 1u);
                if (!ok) return;
                if constexpr (Q4) {
                    constexpr uint32_t D = (SLOT & 1u) * TI_D_COLS, idesc = ti_idesc(16);
                    if (j >= 2) ok = ts_wait(d_empty + 8u * (SLOT & 1u), ((j >> 1) - 1u) & 1u);
                    if (!ok) return;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) ti_mma(tmem + D + 16u * i, tmem + A + 8u * i, b + (i >> 2) * 128u + 2u * (i & 3u), idesc);
                    ti_mma(tmem + D + 128u, tmem + A + 64u, b + 256u, idesc);
                    ti_mma(tmem + D + 144u, tmem + A + 64u, b + 258u, idesc);
                    tm_commit(d_full + 8u * (SLOT & 1u));
                } else {
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        constexpr uint32_t id32 = ti_idesc(32), id16 = ti_idesc(16);
                        const uint32_t D = h * TI_D_COLS;
                        if (j >= 1) ok = ok && ts_wait(d_empty + 8u * h, (j - 1u) & 1u);
                        if (!ok) return;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) ti_mma(tmem + D + 32u * i, tmem + A + 32u * h + 8u * i, b + h * 256u + 2u * i, id32);
                        ti_mma(tmem + D + 128u, tmem + A + 64u + 8u * h, b + 512u, id16);
                        ti_mma(tmem + D + 144u, tmem + A + 64u + 8u * h, b + 514u, id16);
                        tm_commit(d_full + 8u * h);
                    }
                }
                tm_commit(ab_empty + 8u * SLOT);
            };
            for (uint32_t j = 0; j < (uint32_t)n_slabs && ok; j += 4) {
                issue(std::integral_constant<uint32_t, 0>(), j);
                if (j + 1 < (uint32_t)n_slabs) issue(std::integral_constant<uint32_t, 1>(), j + 1);
                if (j + 2 < (uint32_t)n_slabs) issue(std::integral_constant<uint32_t, 2>(), j + 2);
                if (j + 3 < (uint32_t)n_slabs) issue(std::integral_constant<uint32_t, 3>(), j + 3);
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        err_code = 48;
        __syncwarp();
    } else {
        const int group = (warp >> 2) & 1, q = warp & 3;
        const int r = 32 * q + lane;
        const int fr = loose ? (r >> 4) + 8 * (r & 15) : r;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16);
        int tile = u0 / KS;  // of the slab at hand
        uint32_t row_at = (uint32_t)r * SL::PITCH, row_phase = 0, row_mask = 15u;
        auto find_row = [&](int tl) {  // (as in gemm_ts.cu)
            const TsTile t = work.tile(p, tl);
            const TsJob &jb = p.jobs[t.job];
            const int rest0 = jb.F & ~7, f = t.f0 + fr;
            const uintptr_t at = (uintptr_t)jb.w + (size_t)(t.w_row0 + fr) * p.row_bytes;
            const bool rest = f >= rest0 && f < jb.F;
            row_at = (uint32_t)(rest ? TS_ROWS + f - rest0 : r) * SL::LOOSE_PITCH;
            row_mask = rest ? 3u : 15u;
            row_phase = (uint32_t)at & row_mask;
        };
        auto row_of = [&](int j) -> const uint8_t * {
            const uint8_t *rowp = ring + ((uint32_t)j & (R - 1u)) * SLAB + row_at;
            if constexpr (!Q4) rowp += (row_phase + (uint32_t)((u0 + j - tile * KS) * SL::BYTES)) & row_mask;
            return rowp;
        };
        if (loose && n_slabs > 0) find_row(tile);

        if (warp < TI_CONV) {
            // ------------------------------ converters ------------------------------
#pragma unroll 1
            for (int j = group; j < n_slabs && ok; j += 2) {
                if (u0 + j >= (tile + 1) * KS) {
                    tile = (u0 + j) / KS;
                    if (loose) find_row(tile);
                }
                const uint32_t rs = (uint32_t)j & (R - 1u);
                ok = ts_wait(raw_full + 8u * rs, ((uint32_t)j >> p.raw_shift) & 1u);
                struct Emit {
                    bool &ok;
                    uint32_t to, bar, parity;
                    bool wait;
                    __device__ __forceinline__ void operator()(int h, const uint32_t (&o)[32]) const {
                        if (h == 0) {
                            if (ok && wait) ok = ts_wait(bar, parity);  // the slot's previous MMAs
                            ok = __all_sync(0xffffffffu, ok);
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        if (ok) ts_st32(to + 32u * (uint32_t)h, o);
                    }
                    __device__ __forceinline__ void corrections(const uint32_t (&c)[16]) const {
                        if (ok) ts_st16(to + 64u, c);
                    }
                };
                const uint32_t prev = (uint32_t)j - 2u;
                const Emit emit{ok, lanes + TI_A0 + (uint32_t)group * TI_A_COLS, ab_empty + 8u * (prev & (TI_B_SLOTS - 1)), (prev >> 2) & 1u, j >= 2};
                auto done = [&] {
                    __syncwarp();
                    if (lane == 0) tm_mbar_arrive(raw_empty + 8u * rs);
                };
                if constexpr (Q4) ti_conv_q4k(row_of(j), done, emit);
                else ti_conv_q6k<!LOOSE>(row_of(j), (uint32_t)((u0 + j - tile * KS) * SL::BYTES) & 15u, done, emit);
                if (!ok) break;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tm_mbar_arrive(a_full + 8u * group);
            }
            err_code = 49;
        } else {
            // ------------------------------ scalers ------------------------------
            asm volatile("griddepcontrol.wait;" ::: "memory");
            float acc[2][8];
            uint32_t segs = 0;
            for (int u = u0; u < u1 && ok;) {
                tile = u / KS;
                const int u_hi = min((tile + 1) * KS, u1);
                const TsTile t = work.tile(p, tile);
                const TsJob &jb = p.jobs[t.job];
                if (loose) find_row(tile);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[i >> 3][i & 7] = 0.0f;
#pragma unroll 1
                for (int j = u - u0; j < u_hi - u0 && ok; ++j) {
                    if (Q4 && (j & 1) != group) continue;
                    const uint32_t rs = (uint32_t)j & (R - 1u);
                    ok = ts_wait(raw_full + 8u * rs, ((uint32_t)j >> p.raw_shift) & 1u);
                    // d, dmin and the 6-bit scales, or d and this half's eight scales
                    const uint8_t *rowp = row_of(j);
                    float d, dm = 0.0f;
                    uint32_t sc[2];
                    if constexpr (Q4) {
                        const uint4 hdr = *(const uint4 *)rowp;
                        d = half_bits_to_float((uint16_t)hdr.x);
                        dm = half_bits_to_float((uint16_t)(hdr.x >> 16));
                        sc[0] = hdr.y & 0x3F3F3F3Fu;
                        sc[1] = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
                    } else {
                        tm_lds_words<2>(rowp + 192 + 8 * group, sc);
                        d = half_bits_to_float(*(const uint16_t *)(rowp + 208));
                    }
                    __syncwarp();
                    if (lane == 0) tm_mbar_arrive(raw_empty + 8u * rs);
                    // The tokens' block scales come with the activation tile: byte 320 of 384, in the last box (128-byte swizzle).  Read from
                    // memory here they were a trip to L2 in every slab, and what bounded the scalers: 16 x 4096 x 14336 Q4_K 19.5 -> 15.0 us,
                    // 8 x 4096 x 28672 30.7 -> 27.1, Q6_K 8 x 4096 x 14336 27.4 -> 23.7, MoE of 16 tokens 238 -> 218.
                    const uint32_t slot = (uint32_t)j & (TI_B_SLOTS - 1);
                    const uint8_t *dx = smem_raw + (tile_base + slot * B_BYTES + (Q4 ? 4096u : 8192u) - raw_addr);
                    if (ok) ok = ts_wait(b_full + 8u * slot, ((uint32_t)j >> 2) & 1u);
                    if (ok) ok = ts_wait(d_full + 8u * group, (Q4 ? (uint32_t)j >> 1 : (uint32_t)j) & 1u);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t from = lanes + (uint32_t)group * TI_D_COLS;
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {  // eight tokens at a time
                        if (8 * hh >= t.t_count) break;
                        float dxv[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) dxv[i] = *(const float *)(dx + (8 * hh + i) * 128 + ((4 ^ i) << 4));
                        int sum[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) sum[i] = 0;
#pragma unroll
                        for (int s0 = 0; s0 < 8; s0 += 4) {
                            int v[4][8];
#pragma unroll
                            for (int s = 0; s < 4; ++s) ti_ld8(from + 16u * (uint32_t)(s0 + s) + 8u * hh, v[s]);
                            ti_wait_ld();
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                const uint32_t byte = sc[s0 >> 2] >> (8 * s);
                                const int scale = Q4 ? (int)(byte & 0xFFu) : (int)(int8_t)byte;
#pragma unroll
                                for (int i = 0; i < 8; ++i) sum[i] += scale * v[s][i];
                            }
                        }
                        int lo[8], hi[8];
                        ti_ld8(from + 128u + 8u * hh, lo);
                        ti_ld8(from + 144u + 8u * hh, hi);
                        ti_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int corr = lo[i] + 64 * hi[i];
                            if constexpr (Q4)
                                acc[hh][i] = fmaf(dxv[i], __fsub_rn(__fmul_rn(d, (float)sum[i]), __fmul_rn(dm, (float)corr)), acc[hh][i]);
                            else
                                acc[hh][i] = fmaf(dxv[i], __fmul_rn(d, (float)(sum[i] - 32 * corr)), acc[hh][i]);
                        }
                    }
                    // (Behind the last operations: given back ahead of them, as soon as the sums are read, Q6_K of 7 x 4608 x 4096 took 13.0 instead
                    // of 12.5 us, MoE of 24 tokens with a Q6_K down projection 63.7 instead of 62.5, Q4_K of 12 x 3072 x 1024 7.94 instead of 7.84.)
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        tm_mbar_arrive(d_empty + 8u * group);
                        tm_mbar_arrive(dx_read + 8u * slot);
                    }
                }
                if (!ok) break;
                // ---- the tile's part is complete: group 1's sums go to group 0 ----
                if (group == 1) {
                    if (segs >= 1) ok = ts_wait(seg_free, (segs - 1u) & 1u);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
#pragma unroll
                    for (int c = 0; c < 16; ++c) sums[c * TS_ROWS + r] = acc[c >> 3][c & 7];
                    __syncwarp();
                    if (lane == 0) tm_mbar_arrive(seg_full);
                    ++segs;
                    u = u_hi;
                    continue;
                }
                ok = ts_wait(seg_full, segs & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
#pragma unroll
                for (int c = 0; c < 16; ++c) acc[c >> 3][c & 7] += sums[c * TS_ROWS + r];
                __syncwarp();
                if (lane == 0) tm_mbar_arrive(seg_free);
                ++segs;
                const bool live = fr < t.rows;
                const int f = t.f0 + fr;
                const float bias = (live && jb.bias != nullptr) ? jb.bias[f] : 0.0f;
                float *outp = jb.out + (size_t)t.t_row0 * jb.ldo + f;
                const int u_lo = u;
                u = u_hi;
                if (split > 1) {
#pragma unroll
                    for (int c = 0; c < 16; ++c) shared_share[c * TS_ROWS + r] = acc[c >> 3][c & 7];
                    continue;
                }
                if (u_hi - u_lo != KS) {
                    // a share of a cut tile (as in gemm_ts.cu)
                    const uint32_t which = u_lo == u0 ? 0u : 1u;
                    float *mine = p.partial + (size_t)(cta * 2 + (int)which) * (TS_ROWS * TI_COLS) + r;
#pragma unroll
                    for (int c = 0; c < 16; ++c) __stcg(mine + c * TS_ROWS, acc[c >> 3][c & 7]);
                    __threadfence();
                    __syncwarp();
                    if (lane == 0) tm_mbar_arrive(share_bar + 8u * which);
                    // Whoever draws the last ticket adds the shares up when its range is done: drawn and added here, by these four warps, they
                    // kept the sums of the slabs behind waiting (MoE of 16 tokens 206 -> 200 us, FFN input of 8 98.3 -> 94.7).
                    if (warp == TI_CONV) {
                        ok = ts_wait(share_bar + 8u * which, 0u);
                        ok = __all_sync(0xffffffffu, ok);
                        if (lane == 0 && ok) {
                            int *ctr = p.counters + cut_first[which];
                            if (atomicAdd(ctr, 1) == cut_last[which] - cut_first[which]) {
                                *ctr = 0;  // ready for the next launch
                                cut_tile[which] = tile;
                            }
                        }
                        __syncwarp();
                        if (!ok) break;
                    }
                    continue;
                }
                if (live) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        if (c < t.t_count) outp[(size_t)c * jb.ldo] = acc[c >> 3][c & 7] + bias;
                }
            }
            err_code = 50;
        }
    }
    if (!ok) {
        if (lane == 0) atomicExch(p.err, err_code);
        abort_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (abort_flag) {  // bulk copies may still be landing: give them time
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (split > 1) {
        __syncwarp();
        ts_cluster_sync();  // the shares of the split tile are complete
        const TsTile t = work.tile(p, cta / split);
        const TsJob &jb = p.jobs[t.job];
        const int part = cta - cta / split * split, c_lo = t.t_count * part / split, c_hi = t.t_count * (part + 1) / split;
        const int r = threadIdx.x & (TS_ROWS - 1), fr = loose ? (r >> 4) + 8 * (r & 15) : r, f = t.f0 + fr;
        if (threadIdx.x >= 256 && threadIdx.x < 512 && fr < t.rows) {  // (the scalers: they have waited for the kernel ahead)
            const float bias = jb.bias != nullptr ? jb.bias[f] : 0.0f;
            for (int c = c_lo + (int)((threadIdx.x - 256) >> 7); c < c_hi; c += 2) {
                float v[TS_MAX_SPLIT];
#pragma unroll
                for (int i = 0; i < TS_MAX_SPLIT; ++i) {
                    v[i] = 0.0f;
                    if (i < split)
                        asm volatile("ld.shared::cluster.f32 %0, [%1];"
                                     : "=f"(v[i]) : "r"(ts_mapa(share_addr + 4u * (uint32_t)(c * TS_ROWS + r), (uint32_t)i)) : "memory");
                }
                float sum = v[0];
#pragma unroll
                for (int i = 1; i < TS_MAX_SPLIT; ++i)
                    if (i < split) sum += v[i];
                jb.out[(size_t)(t.t_row0 + c) * jb.ldo + f] = sum + bias;
            }
        }
        __syncwarp();
        ts_cluster_sync();  // nobody leaves while its share is being read
    }
    // Shares of cut tiles, in the order of K (the scalers: they have waited for the kernel ahead).  (Plans without cut tiles pass by without
    // looking: 8 x 2048 x 2048 Q4_K 7.5 -> 7.25 us.)
    for (int s = 0; s < 2 && split == 1 && !p.whole; ++s) {
        const int tile = cut_tile[s];
        if (tile < 0 || threadIdx.x < 256 || threadIdx.x >= 512) continue;
        __threadfence();
        const TsTile t = work.tile(p, tile);
        const TsJob &jb = p.jobs[t.job];
        const int first = cut_first[s], last = cut_last[s], slot0 = cut_slot[s];
        const int r = threadIdx.x & (TS_ROWS - 1), fr = loose ? (r >> 4) + 8 * (r & 15) : r, f = t.f0 + fr;
        const int c0 = 8 * (int)((threadIdx.x - 256) >> 7);  // eight of the tokens
        if (fr >= t.rows || c0 >= t.t_count) continue;
        float acc[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = 0.0f;
#pragma unroll 4
        for (int k = first; k <= last; ++k) {  // (the ranges behind the first one start inside the tile)
            const float *from = p.partial + (size_t)(k * 2 + (k == first ? slot0 : 0)) * (TS_ROWS * TI_COLS) + c0 * TS_ROWS + r;
            float v[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = __ldcg(from + c * TS_ROWS);
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[c] += v[c];
        }
        const float bias = jb.bias != nullptr ? jb.bias[f] : 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (c0 + c < t.t_count) jb.out[(size_t)(t.t_row0 + c0 + c) * jb.ldo + f] = acc[c] + bias;
    }
    if (warp == TI_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// ---- host ----
static int ti_planes(int kind) { return kind == KIND_Q6_K ? 2 : 1; }

size_t gemm_ti_xq_bytes(int kind, int rows, int K) { return (size_t)ti_planes(kind) * rows * ((K + QK_K - 1) / QK_K) * 384; }

bool gemm_ti_supported(int kind, const void *W, int K, int F) {
    return (kind == KIND_Q4_K || kind == KIND_Q6_K) && gemm_ts_supported(kind, W, 1, K, F);
}

template <int KIND, bool LOOSE>
static cudaError_t ti_launch(const TsMaps &maps, TsParams &p, int n_cta, int dev, cudaStream_t s) {
    const int fixed = 16 + 512 + 1024 + TI_B_SLOTS * (int)ti_b_bytes<KIND>() + 2 * TI_COLS * TS_ROWS * 4;
    const int slab = ts_slab_bytes<KIND>(LOOSE);
    constexpr int MOST = 224 * 1024;
    p.raw_shift = fixed + 8 * slab <= MOST ? 3 : 2;
    const int smem = fixed + (slab << p.raw_shift);
    static std::atomic<uint64_t> configured{0};
    const bool known = dev >= 0 && dev < 64;
    if (!known || !(configured.load(std::memory_order_relaxed) >> dev & 1)) {
        if (cudaError_t e = cudaFuncSetAttribute(gemm_ti_kernel<KIND, LOOSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST)) return e;
        if (known) configured.fetch_or((uint64_t)1 << dev, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_cta, 1, 1);
    cfg.blockDim = dim3(TI_THREADS, 1, 1);
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
    return cudaLaunchKernelEx(&cfg, gemm_ti_kernel<KIND, LOOSE>, maps, p);
}
static cudaError_t ti_dispatch(int kind, const TsMaps &maps, TsParams &p, int n_cta, int dev, cudaStream_t s) {
    if (kind == KIND_Q4_K) return ti_launch<KIND_Q4_K, false>(maps, p, n_cta, dev, s);
    return p.loose ? ti_launch<KIND_Q6_K, true>(maps, p, n_cta, dev, s) : ti_launch<KIND_Q6_K, false>(maps, p, n_cta, dev, s);
}
static cudaError_t ti_encode_x(int kind, CUtensorMap *m, const uint8_t *xq, int rows, int nb) {
    return ts_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, xq, (cuuint64_t)nb * 384, (cuuint64_t)rows * ti_planes(kind), (cuuint64_t)nb * 384, 128,
                     TI_COLS, CU_TENSOR_MAP_SWIZZLE_128B);
}

cudaError_t launch_gemm_ti(int kind, const GemvJobSpec *jobs, int n_jobs, const uint8_t *xq, int T, int K, float *partial,
                           int *counters, int *err_flag, cudaStream_t s) {
    if (n_jobs < 1 || n_jobs > TS_MAX_JOBS || T < 1) return cudaErrorInvalidValue;
    TsParams p;
    TsMaps maps;
    memset(&p, 0, sizeof(p));
    p.nb = p.slabs = (K + QK_K - 1) / QK_K;
    p.row_bytes = (long)p.nb * block_bytes(kind);
    p.partial = partial;
    p.counters = counters;
    p.err = err_flag;
    p.n_jobs = n_jobs;
    p.T = T;
    p.t_tiles = (T + TI_COLS - 1) / TI_COLS;
    int row_tiles = 0;
    for (int j = 0; j < n_jobs; ++j) p.loose |= ts_loose(kind, jobs[j].W, p.row_bytes);
    for (int j = 0; j < n_jobs; ++j) {
        p.jobs[j] = TsJob{(const uint8_t *)jobs[j].W, jobs[j].out, jobs[j].bias, jobs[j].F, jobs[j].ldo, row_tiles};
        row_tiles += (jobs[j].F + TS_ROWS - 1) / TS_ROWS;
        if (cudaError_t e = ts_encode_weights(kind, &maps.w[j], jobs[j].W, p.row_bytes, (size_t)jobs[j].F, p.loose != 0)) return e;
    }
    p.tiles = row_tiles * p.t_tiles;
    if (cudaError_t e = ti_encode_x(kind, &maps.x, xq, T, p.nb)) return e;
    int dev;
    const TsPlan pl = ti_plan(kind, p.tiles, p.slabs, device_sm_count(&dev));
    p.split = pl.split;
    p.whole = pl.whole;
    return ti_dispatch(kind, maps, p, pl.n_cta, dev, s);
}

cudaError_t launch_gemm_ti_grouped(int kind, const GemvJobSpec *jobs, int n_jobs, int n_groups, const uint8_t *xq,
                                   int total_rows, int K, const int *group_counts, const int *group_offsets, float *partial,
                                   int *counters, int *err_flag, cudaStream_t s) {
    if (n_groups <= 0 || total_rows <= 0) return cudaSuccess;
    if (n_jobs < 1 || n_jobs > TS_MAX_JOBS || n_groups > TS_MAX_GROUPS) return cudaErrorInvalidValue;
    TsParams p;
    TsMaps maps;
    if (cudaError_t e = ts_grouped_params(kind, jobs, n_jobs, n_groups, total_rows, K, group_counts, group_offsets, p, maps))
        return e;
    p.bn = TI_COLS;
    p.partial = partial;
    p.counters = counters;
    p.err = err_flag;
    if (cudaError_t e = ti_encode_x(kind, &maps.x, xq, total_rows, p.nb)) return e;
    int dev;
    const int sms = device_sm_count(&dev);
    return ti_dispatch(kind, maps, p, sms, dev, s);
}

}  // namespace mcu

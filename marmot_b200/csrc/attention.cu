// Attention over a paged f16 pool with one warp per (token, KV head, chunk of 128 positions).
//
// The arithmetic is that of paged_attention_mma_kernel (decoder.cu): four tiles of 32 positions, scores and P V on mma.sync with Q and P
// split into f16 head and tail, the four tiles' softmax states merged in order, the chunks' states merged in chunk order.  Results
// are the same bit for bit; what differs is who does it and how the tiles come:
//
// - K and V tiles are TMA boxes (64 dimensions x up to 32 rows of one pool block, 128-byte swizzle, which ldmatrix reads without bank
//   conflicts).  Sixteen cp.async per lane and tile kept a warp's issue slot 2200 of the 10000 cycles that a chunk took.
// - One warp does all four tiles of a chunk: the states are merged in registers, no barrier and no trip through shared memory
//   (1600 cycles of the 10000).
// - Decode steps (attention_decode_kernel): persistent, chunk x of the list of all chunks to warp x % warps, every warp with its own
//   ring of tiles, so the next tiles are on their way under the arithmetic.
// - Prompts (attention_prompt_kernel): a CTA fetches the chunk once for the tokens of its block that stand at consecutive
//   positions of a sequence; every warp takes as many of them as fill the eight rows of A.  A block of short runs (decode steps among
//   prompts) is taken token by token, four warps to a token.
//
// Measured: 64 sequences of 256 to 4096 positions, 8 KV heads of 128 (570 MB): 143 -> 102 us, 5.6 TB/s; a prompt of 500 tokens of the
// same model 119 -> 51.  A warp takes 20000 cycles per chunk of the first (four tiles of 1000 for the scores and 800 for P V, the
// copies' latencies, q, the store), eight warps on an SM: the memory is close behind.
#include "paged_attention.cuh"

#include "gemm_ts_dev.cuh"
#include "kernels.h"

#include <cstdlib>
#include <cstring>

namespace mcu {

constexpr int AT_WARPS = 8;
constexpr int AT_HALF_BYTES = PM_TILE * 128;  // 64 dimensions of a tile's rows
constexpr int AT_RING_BYTES = 24 * 1024;      // of a warp (decode steps)
constexpr int AT_MAX_TOKENS = 256;            // decode steps: the tokens' chunk counts are summed up in shared memory
constexpr int AT_BLOCK = 32;                  // prompts: most tokens of a CTA
constexpr int AT_SHORT = 4;                   // prompts: blocks with runs of fewer tokens on average are taken token by token

struct AttnMaps {
    CUtensorMap k, v;  // [pool block, layer and KV head][64 dimensions][position][dimension]
};

template <int HD>
struct At {
    static constexpr int HALVES = HD / 64, TILE = HALVES * AT_HALF_BYTES, KS = HD / 16, NT = HD / 8, SLOTS = AT_RING_BYTES / TILE;
    static constexpr int Q_BYTES = KS * 32 * 16;  // a warp's A fragments: heads and tails
    static constexpr int PROMPT_TILES = HD == 64 ? 16 : 8;  // of a prompt CTA: K 0..3, V 0..3; token by token two or one per warp
};

__device__ __forceinline__ void at_tma_4d(uint32_t dst, const CUtensorMap *map, int row, int slab, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(0), "r"(row), "r"(0), "r"(slab), "r"(bar) : "memory");
}
// Where row r of a tile lies, and how far its next 64 dimensions: boxes of `1 << shift` rows, one per pool block, each [64
// dimensions][row][128 bytes], swizzled by the 128-byte line (at least eight rows, or the lines are those of smaller boxes).
template <int HD>
struct AtRows {
    int shift;
    __device__ __forceinline__ uint32_t row(int r) const { return (uint32_t)((((r >> shift) << shift) * At<HD>::HALVES + (r & ((1 << shift) - 1))) * 128); }
    __device__ __forceinline__ uint32_t piece(int r, int pc) const {
        const uint32_t line = row(r) + (uint32_t)((pc >> 3) << (shift + 7));
        return line + ((((uint32_t)pc & 7u) ^ ((line >> 7) & 7u)) << 4);
    }
    __device__ __forceinline__ uint32_t value(int r, int d) const { return piece(r, d >> 3) + (uint32_t)(d & 7) * 2u; }
};

// The pool blocks of a chunk, block i in lane i (at least four positions to a block; smaller ones are looked up tile by tile).
__device__ __forceinline__ uint32_t at_blocks(const PagedParams &p, uint32_t seq, uint32_t len, uint32_t p0, int lane) {
    const uint32_t pos = p0 + ((uint32_t)lane << p.block_shift), lb = pos >> p.block_shift;
    if (lane > 0 && ((uint32_t)lane << p.block_shift) >= PM_CHUNK) return 0xFFFFFFFFu;
    return pos < len && lb < (uint32_t)p.max_blocks ? __ldg(p.table + (size_t)seq * p.max_blocks + lb) : 0xFFFFFFFFu;
}
// Ask for tile w of a chunk (positions p0 + 32 w ..) of a sequence whose context is `len`: one box per pool block, one lane each.
// Returns the rows that hold data: blocks that the table maps, positions inside the context.
template <int HD>
__device__ __forceinline__ uint32_t at_load_tile(const PagedParams &p, const CUtensorMap *map, uint32_t blocks, uint32_t len, int h, uint32_t p0,
                                                 int w, uint32_t dst, uint32_t bar, int lane, uint32_t seq) {
    const int shift = min(p.block_shift, 5), n = PM_TILE >> shift;
    const uint32_t k0 = p0 + (uint32_t)(w * PM_TILE);
    const uint32_t in_chunk = (uint32_t)(w * PM_TILE) + ((uint32_t)lane << shift);  // first position of this lane's box
    uint32_t tb = __shfl_sync(0xffffffffu, blocks, (int)(in_chunk >> p.block_shift) & 31);
    if (p.block_shift < 2) {
        const uint32_t lb = (p0 + in_chunk) >> p.block_shift;
        tb = lane < n && p0 + in_chunk < len && lb < (uint32_t)p.max_blocks ? __ldg(p.table + (size_t)seq * p.max_blocks + lb) : 0xFFFFFFFFu;
    }
    const bool mine = lane < n && tb != 0xFFFFFFFFu && p0 + in_chunk < len;
    const uint32_t have = __ballot_sync(0xffffffffu, mine);
    // (the bytes may arrive ahead of their announcement: the phase ends with lane 0's arrival at the earliest)
    if (lane == 0) tm_mbar_expect_tx(bar, (uint32_t)__popc(have) * (uint32_t)(HD * 2 << shift));
    if (mine) {
        const int slab = (int)((tb * (uint32_t)p.n_layers + (uint32_t)p.layer) * (uint32_t)p.n_kv_heads + (uint32_t)h);
        at_tma_4d(dst + (uint32_t)(lane * HD * 2 << shift), map, (int)((p0 + in_chunk) & ((1u << p.block_shift) - 1u)), slab, bar);
    }
    const uint32_t inside = len - k0 >= 32u ? 0xffffffffu : (1u << (len - k0)) - 1u;  // (len > k0)
    if (have == (n >= 32 ? 0xffffffffu : (1u << n) - 1u)) return inside;
    return __ballot_sync(0xffffffffu, ((have >> (lane >> shift)) & 1u) != 0) & inside;
}
// Rows without data of a V tile: never scored, but 0 * garbage must not become NaN.
template <int HD>
__device__ __forceinline__ void at_zero_rows(const AtRows<HD> &rows, uint32_t tile, uint32_t live, int lane) {
    for (int idx = lane; idx < PM_TILE * (HD / 8); idx += 32) {
        const int row = idx / (HD / 8), pc = idx % (HD / 8);
        if (!((live >> row) & 1u))
            asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(tile + rows.piece(row, pc)), "r"(0u) : "memory");
    }
}

// A fragments of Q into this lane's part of `qf`: row g of A (of this lane) is `qrow` (null: zeros), rotated when there is a table.
// a0 = dimensions 16 s + 2 tq, + 1; a2 = dimensions 16 s + 8 + 2 tq, + 1.
template <int HD>
__device__ __forceinline__ void at_load_q(const float *qrow, const float2 *rope, int neox, float scale, uint4 *qf, int lane) {
    constexpr int KS = At<HD>::KS;
    const int tq = lane & 3;
    float2 qv[KS][2];
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int hk = 0; hk < 2; ++hk)
            qv[s][hk] = qrow != nullptr ? *(const float2 *)(qrow + 16 * s + 8 * hk + 2 * tq) : make_float2(0.0f, 0.0f);
    if (rope != nullptr) {
        if (!neox) {  // the pair (d, d + 1) is one float2
            float2 cs[KS][2];
#pragma unroll
            for (int s = 0; s < KS; ++s)
#pragma unroll
                for (int hk = 0; hk < 2; ++hk) cs[s][hk] = __ldg(rope + ((16 * s + 8 * hk + 2 * tq) >> 1));
#pragma unroll
            for (int s = 0; s < KS; ++s)
#pragma unroll
                for (int hk = 0; hk < 2; ++hk) {
                    const float x = qv[s][hk].x, y = qv[s][hk].y, c = cs[s][hk].x, sn = cs[s][hk].y;
                    qv[s][hk].x = __fsub_rn(__fmul_rn(x, c), __fmul_rn(y, sn));
                    qv[s][hk].y = __fadd_rn(__fmul_rn(x, sn), __fmul_rn(y, c));
                }
        } else {  // the pairs (d, d +- HD/2): the partner of k step s is k step s +- KS/2 of this same lane
            float4 cs[KS / 2][2];
#pragma unroll
            for (int s = 0; s < KS / 2; ++s)
#pragma unroll
                for (int hk = 0; hk < 2; ++hk) cs[s][hk] = __ldg((const float4 *)(rope + 16 * s + 8 * hk + 2 * tq));
#pragma unroll
            for (int s = 0; s < KS / 2; ++s)
#pragma unroll
                for (int hk = 0; hk < 2; ++hk) {
                    const float2 lo = qv[s][hk], hi = qv[s + KS / 2][hk];
                    const float4 c = cs[s][hk];
                    qv[s][hk].x = __fsub_rn(__fmul_rn(lo.x, c.x), __fmul_rn(hi.x, c.y));
                    qv[s][hk].y = __fsub_rn(__fmul_rn(lo.y, c.z), __fmul_rn(hi.y, c.w));
                    qv[s + KS / 2][hk].x = __fadd_rn(__fmul_rn(lo.x, c.y), __fmul_rn(hi.x, c.x));
                    qv[s + KS / 2][hk].y = __fadd_rn(__fmul_rn(lo.y, c.w), __fmul_rn(hi.y, c.z));
                }
        }
    }
#pragma unroll
    for (int s = 0; s < KS; ++s) {
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int hk = 0; hk < 2; ++hk) {
            float x = qv[s][hk].x, y = qv[s][hk].y;
            if (scale != 1.0f) {
                x = __fmul_rn(x, scale);
                y = __fmul_rn(y, scale);
            }
            split_half2(x, y, hi[hk], lo[hk]);
        }
        qf[32 * s + lane] = make_uint4(hi[0], lo[0], hi[1], lo[1]);
    }
}

// Scores of a tile and their softmax: P as f16 heads and tails (the A fragments of P V), the row's maximum and sum.
template <int HD>
__device__ __forceinline__ void at_scores(const AtRows<HD> &rows, uint32_t tile, const uint4 *qf, uint32_t row_live, int lane, uint32_t (&phi)[4], uint32_t (&plo)[4],
                                          float &m, float &l) {
    const int tq = lane & 3;
    float sc[4][4], st[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[j][e] = st[j][e] = 0.0f;
#pragma unroll
    for (int s = 0; s < At<HD>::KS; s += 2) {
        const uint4 qa = qf[32 * s + lane], qb = qf[32 * (s + 1) + lane];
        uint32_t b[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            // matrices: (keys 8j.., piece 2s), (piece 2s+1), (piece 2s+2), (piece 2s+3)
            ldsm_x4(tile + rows.piece(8 * j + (lane & 7), 2 * s + (lane >> 3)), b[j][0], b[j][1], b[j][2], b[j][3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_hi_lo(sc[j], qa.x, qa.y, qa.z, qa.w, b[j][0], b[j][1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_hi_lo(st[j], qb.x, qb.y, qb.z, qb.w, b[j][2], b[j][3]);
    }
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        sc[j][0] = (sc[j][0] + st[j][0]) + (sc[j][2] + st[j][2]);
        sc[j][1] = (sc[j][1] + st[j][1]) + (sc[j][3] + st[j][3]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (!((row_live >> (8 * j + 2 * tq + e)) & 1u)) sc[j][e] = -INFINITY;
            mx = fmaxf(mx, sc[j][e]);
        }
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    float psum = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float w0 = mx == -INFINITY ? 0.0f : expf(sc[j][0] - mx);
        const float w1 = mx == -INFINITY ? 0.0f : expf(sc[j][1] - mx);
        psum += w0 + w1;
        split_half2(w0, w1, phi[j], plo[j]);
    }
    psum += __shfl_xor_sync(0xffffffffu, psum, 1);
    psum += __shfl_xor_sync(0xffffffffu, psum, 2);
    m = mx;
    l = psum;
}

// acc += e * (P V) of a tile, eight dimension tiles at a time.
template <int HD>
__device__ __forceinline__ void at_pv(const AtRows<HD> &rows, uint32_t tile, const uint32_t (&phi)[4], const uint32_t (&plo)[4], float e, int lane,
                                      float (&acc)[At<HD>::NT][2]) {
    const int mi = lane >> 3;
#pragma unroll
    for (int n0 = 0; n0 < At<HD>::NT; n0 += 8) {
        float o[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.0f;
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int n = 0; n < 8; n += 4) {
                // matrices: (keys 16u.., piece n), (keys 16u+8.., piece n), (keys 16u.., piece n+1), (keys 16u+8.., piece n+1)
                const int r = 16 * u + 8 * (mi & 1) + (lane & 7);
                uint32_t b[2][4];
#pragma unroll
                for (int h2 = 0; h2 < 2; ++h2)
                    ldsm_x4_trans(tile + rows.piece(r, n0 + n + 2 * h2 + (mi >> 1)), b[h2][0], b[h2][1], b[h2][2], b[h2][3]);
#pragma unroll
                for (int h2 = 0; h2 < 2; ++h2) {
                    mma_hi_lo(o[n + 2 * h2], phi[2 * u], plo[2 * u], phi[2 * u + 1], plo[2 * u + 1], b[h2][0], b[h2][1]);
                    mma_hi_lo(o[n + 2 * h2 + 1], phi[2 * u], plo[2 * u], phi[2 * u + 1], plo[2 * u + 1], b[h2][2], b[h2][3]);
                }
            }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            acc[n0 + n][0] += (o[n][0] + o[n][2]) * e;
            acc[n0 + n][1] += (o[n][1] + o[n][3]) * e;
        }
    }
}

// What the scores of a chunk's four tiles leave behind.  push() after every tile (of the four, present or not), weigh() after the
// fourth; pop() then gives them back in order.  A shift register, so that the loops over the tiles can stay loops: unrolled, the
// kernels' code took 27 us to come through the instruction cache with the first chunk of every launch (17 rolled, and 150 -> 107
// for the whole).
struct AtTiles {
    uint32_t phi[4][4], plo[4][4];
    float m[4], l[4];  // l: the tiles' weights after weigh()
    __device__ __forceinline__ void shift() {
#pragma unroll
        for (int w = 3; w > 0; --w) {
#pragma unroll
            for (int i = 0; i < 4; ++i) phi[w][i] = phi[w - 1][i], plo[w][i] = plo[w - 1][i];
            m[w] = m[w - 1], l[w] = l[w - 1];
        }
    }
    __device__ __forceinline__ void push() { shift(), m[0] = -INFINITY, l[0] = 0.0f; }
    // the tiles' weights in the chunk's state, and that state's maximum and sum
    __device__ __forceinline__ void weigh(float &M, float &L) {
        M = -INFINITY;
#pragma unroll
        for (int w = 0; w < 4; ++w) M = fmaxf(M, m[w]);
        L = 0.0f;
#pragma unroll
        for (int w = 3; w >= 0; --w) {  // the order of the positions
            const float e = (M == -INFINITY || m[w] == -INFINITY) ? 0.0f : expf(m[w] - M);
            L += l[w] * e;
            l[w] = e;
        }
    }
};
// Row g of the chunk's state: the result when it is the token's only chunk, a partial state otherwise.
template <int HD>
__device__ __forceinline__ void at_store(const PagedParams &p, float *partial, int n_chunks, size_t row, int c, bool only, float M, float L, int tq,
                                         const float (&acc)[At<HD>::NT][2]) {
    if (only) {
        float *to = p.out + row * HD;
#pragma unroll
        for (int n = 0; n < At<HD>::NT; ++n) {
            to[8 * n + 2 * tq] = L > 0.0f ? acc[n][0] / L : 0.0f;
            to[8 * n + 2 * tq + 1] = L > 0.0f ? acc[n][1] / L : 0.0f;
        }
        return;
    }
    float *pr = partial + (row * n_chunks + c) * (HD + 2);
    if (tq == 0) *(float2 *)pr = make_float2(M, L);
#pragma unroll
    for (int n = 0; n < At<HD>::NT; ++n) *(float2 *)(pr + 2 + 8 * n + 2 * tq) = make_float2(acc[n][0], acc[n][1]);
}

// Decode steps: at most one token per sequence, RoPE of q and the new row's RoPE and append included.
template <int HD>
__global__ void __launch_bounds__(32 * AT_WARPS, 1)
attention_decode_kernel(const __grid_constant__ AttnMaps maps, PagedParams p, int n_chunks, float *partial, FusedDecode fd, int *err) {
    using A = At<HD>;
    extern __shared__ uint8_t at_smem[];
    __shared__ __align__(8) uint64_t bars[AT_WARPS][A::SLOTS];
    __shared__ uint32_t slot_live[AT_WARPS][A::SLOTS];
    __shared__ int scan[AT_WARPS], prefix[AT_MAX_TOKENS + 1];  // chunks of the tokens ahead
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), g = lane >> 2, tq = lane & 3;
    const uint32_t raw = tm_smem_u32(at_smem), base = (raw + 1023u) & ~1023u;
    const uint32_t ring = base + (uint32_t)warp * AT_RING_BYTES;
    uint8_t *ring_ptr = at_smem + (ring - raw);
    uint4 *qf = (uint4 *)(at_smem + (base - raw) + AT_WARPS * AT_RING_BYTES + warp * A::Q_BYTES);
    const uint32_t bar0 = tm_smem_u32(&bars[warp][0]);
    if (lane < A::SLOTS) tm_mbar_init(bar0 + 8u * (uint32_t)lane, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int T = p.n_tokens, H = p.n_kv_heads, gsize = p.n_q_heads / H;
    auto chunks_of = [&](uint32_t len) { return min(n_chunks, (int)((len + (uint32_t)PM_CHUNK - 1u) / (uint32_t)PM_CHUNK)); };
    {
        const int per = (T + 32 * AT_WARPS - 1) / (32 * AT_WARPS), lo = min(T, (int)threadIdx.x * per), hi = min(T, lo + per);
        int mine = 0;
        for (int t = lo; t < hi; ++t) {
            const int n = chunks_of(p.meta[t * 4 + 1] + 1u);
            prefix[t + 1] = n;
            mine += n;
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) scan[warp] = incl;
        __syncthreads();
        int at = incl - mine;
        for (int w = 0; w < warp; ++w) at += scan[w];
        for (int t = lo; t < hi; ++t) prefix[t + 1] = at += prefix[t + 1];
        if (threadIdx.x == 0) prefix[0] = 0;
        __syncthreads();
    }
    // Chunk x of the list (token by token, head by head) goes to warp x % warps: all warps work on the same few sequences at a time.
    // (With a contiguous share of the list each, they touch the whole pool at a time: address translation, 30 us for the first chunks.)
    const int all = prefix[T] * H, n_warps = (int)gridDim.x * AT_WARPS, id = warp * (int)gridDim.x + (int)blockIdx.x;
    const int n_items = id < all ? (all - id + n_warps - 1) / n_warps : 0;
    struct Cursor {
        int t, h, c, n;
        uint32_t seq, len;
    };
    auto item = [&](int i) {
        const int x = id + i * n_warps;
        int lo = 0, hi = T;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid] * H <= x) lo = mid;
            else hi = mid;
        }
        const int in = x - prefix[lo] * H, n = prefix[lo + 1] - prefix[lo];
        return Cursor{lo, in / n, in % n, n, p.meta[lo * 4], p.meta[lo * 4 + 1] + 1u};
    };
    auto tiles_of = [&](const Cursor &x) { return min(4, (int)((x.len - (uint32_t)x.c * PM_CHUNK + PM_TILE - 1u) / PM_TILE)); };

    // the producer's side: tiles K 0.., V 0.. of every chunk, in order
    const AtRows<HD> rows{min(p.block_shift, 5)};
    Cursor prod{0, 0, 0, 1, 0u, 0u};
    uint32_t blocks = 0xFFFFFFFFu;
    int prod_item = 0, prod_tile = 0, prod_slot = 0;
    auto next_item = [&]() {
        prod = item(prod_item);
        blocks = at_blocks(p, prod.seq, prod.len, (uint32_t)prod.c * PM_CHUNK, lane);
        // its q and angles into L1
        const char *qrow = (const char *)(p.q + ((size_t)prod.t * p.n_q_heads + (size_t)prod.h * gsize) * HD);
        const char *rope = (const char *)(fd.rope + (size_t)prod.t * (HD / 2));
        for (int i = lane * 128; i < gsize * HD * 4 + HD * 4; i += 32 * 128)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(i < gsize * HD * 4 ? qrow + i : rope + (i - gsize * HD * 4)));
    };
    if (n_items > 0) next_item();
    auto ask = [&]() {
        if (prod_item == n_items) return;
        const int nt = tiles_of(prod);
        const bool is_v = prod_tile >= nt;
        const uint32_t live = at_load_tile<HD>(p, is_v ? &maps.v : &maps.k, blocks, prod.len, prod.h, (uint32_t)prod.c * PM_CHUNK,
                                               is_v ? prod_tile - nt : prod_tile, ring + (uint32_t)(prod_slot * A::TILE),
                                               bar0 + 8u * (uint32_t)prod_slot, lane, prod.seq);
        if (lane == 0) slot_live[warp][prod_slot] = live;
        __syncwarp();
        if (++prod_slot == A::SLOTS) prod_slot = 0;
        if (++prod_tile == 2 * nt) {
            prod_tile = 0;
            if (++prod_item < n_items) next_item();
        }
    };
#pragma unroll 1
    for (int i = 0; i < A::SLOTS; ++i) ask();

    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    auto release = [&](bool dirty) {  // this lane is done with the slot; dirty: ordinary stores went to it
        if (dirty) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (++slot == A::SLOTS) slot = 0, phase ^= 1u;
        ask();
    };
    for (int i = 0; i < n_items && ok; ++i) {
        const Cursor cons = item(i);
        const int t = cons.t, h = cons.h, c = cons.c, nt = tiles_of(cons);
        const size_t head_row = (size_t)t * p.n_q_heads + (size_t)h * gsize;
        at_load_q<HD>(g < gsize ? p.q + (head_row + g) * HD : nullptr, fd.rope + (size_t)t * (HD / 2), fd.neox, p.scale, qf, lane);
        // The token's own row (position len - 1) comes from k_new / v_new, rotated and rounded to f16, and goes to the pool too (no
        // other warp of the launch uses that pool row: every other position belongs to an earlier step).
        const uint32_t new_pos = cons.len - 1u;
        const bool newest = new_pos / PM_CHUNK == (uint32_t)c;
        const int new_tile = newest ? (int)(new_pos % PM_CHUNK) / PM_TILE : -1, new_row = (int)(new_pos % PM_TILE);
        size_t pool_at = 0;
        if (newest) {
            const uint32_t kv_slot = p.meta[t * 4 + 2];
            const size_t bs = (size_t)1 << p.block_shift, slab = ((size_t)(kv_slot >> p.block_shift) * p.n_layers + p.layer) * H + h;
            pool_at = (slab * bs + (kv_slot & (uint32_t)(bs - 1))) * HD;
        }
        AtTiles tiles;
        float M, L;
#pragma unroll 1
        for (int w = 0; w < 4; ++w) {
            tiles.push();
            if (w >= nt || !ok) continue;
            ok = ts_wait(bar0 + 8u * (uint32_t)slot, phase);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) continue;
            const uint32_t tile = ring + (uint32_t)(slot * A::TILE);
            uint32_t live = slot_live[warp][slot];
            if (w == new_tile) {
                uint8_t *to = ring_ptr + slot * A::TILE;
                const float2 *rope = fd.rope + (size_t)t * (HD / 2);
                const float *krow = p.k_new + ((size_t)t * H + h) * HD;
                for (int k = lane; k < HD / 2; k += 32) {
                    const float cs = rope[k].x, sn = rope[k].y;
                    const int ev = fd.neox ? k : 2 * k, od = fd.neox ? k + HD / 2 : 2 * k + 1;
                    const float xe = krow[ev], xo = krow[od];
                    const __half ke = __float2half_rn(__fsub_rn(__fmul_rn(xe, cs), __fmul_rn(xo, sn)));
                    const __half ko = __float2half_rn(__fadd_rn(__fmul_rn(xe, sn), __fmul_rn(xo, cs)));
                    *(__half *)(to + rows.value(new_row, ev)) = ke;
                    *(__half *)(to + rows.value(new_row, od)) = ko;
                    ((__half *)p.kv_k)[pool_at + ev] = ke;
                    ((__half *)p.kv_k)[pool_at + od] = ko;
                }
                __syncwarp();
            }
            at_scores<HD>(rows, tile, qf, live, lane, tiles.phi[0], tiles.plo[0], tiles.m[0], tiles.l[0]);
            release(w == new_tile);
        }
        tiles.weigh(M, L);
        float acc[A::NT][2];
#pragma unroll
        for (int n = 0; n < A::NT; ++n) acc[n][0] = acc[n][1] = 0.0f;
#pragma unroll 1
        for (int w = 0; w < nt && ok; ++w, tiles.shift()) {
            ok = ts_wait(bar0 + 8u * (uint32_t)slot, phase);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t tile = ring + (uint32_t)(slot * A::TILE), live = slot_live[warp][slot];
            if (live != 0xffffffffu) at_zero_rows<HD>(rows, tile, live, lane);
            if (w == new_tile) {
                __syncwarp();
                uint8_t *to = ring_ptr + slot * A::TILE;
                const float *vrow = p.v_new + ((size_t)t * H + h) * HD;
                for (int d = lane; d < HD; d += 32) {
                    const __half vv = __float2half_rn(vrow[d]);
                    *(__half *)(to + rows.value(new_row, d)) = vv;
                    ((__half *)p.kv_v)[pool_at + d] = vv;
                }
            }
            __syncwarp();
            at_pv<HD>(rows, tile, tiles.phi[3], tiles.plo[3], tiles.l[3], lane, acc);
            release(live != 0xffffffffu || w == new_tile);
        }
        if (ok && g < gsize)
            at_store<HD>(p, partial, n_chunks, head_row + g, c, cons.n == 1, M, L, tq, acc);
    }
    if (!ok) {  // a tile never came: report it, and give the copies under way time to land
        if (lane == 0) atomicExch(err, 60);
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
}

struct AtPromptShared {
    __align__(8) uint64_t bars[AT_WARPS][2];
    uint32_t tile_live[AT_WARPS], seq[AT_BLOCK], pos[AT_BLOCK];
    float m[AT_WARPS][8], l[AT_WARPS][8];
};

// The tokens of a block one by one: group g of four warps takes the tokens g, g + 2 ..; a warp takes a tile of 32 positions of the chunk, and
// the four states are merged through shared memory (as in paged_attention_mma_kernel).  For blocks of short runs: run by run a token costs its CTA 5.5 us, and
// seven warps stand by (64 sequences of 2000 positions with a token each, 8 KV heads of 128: 247 us run by run, 120 so).
template <int HD>
__device__ __forceinline__ bool at_tokens(const AttnMaps &maps, const PagedParams &p, int t_lo, int n_tok, int h, int c, int n_chunks, float *partial,
                                          uint32_t base, uint4 *qf_all, AtPromptShared &sh) {
    using A = At<HD>;
    constexpr bool BOTH = A::PROMPT_TILES == 2 * AT_WARPS;  // a slot for K and one for V
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3, group = warp >> 2, wl = warp & 3;
    const int gsize = p.n_q_heads / p.n_kv_heads;
    const AtRows<HD> rows{min(p.block_shift, 5)};
    const uint32_t tile_k = base + (uint32_t)(warp * (BOTH ? 2 : 1) * A::TILE), tile_v = BOTH ? tile_k + (uint32_t)A::TILE : tile_k;
    const uint32_t bar = tm_smem_u32(&sh.bars[warp][0]), p0 = (uint32_t)c * PM_CHUNK;
    uint4 *qf = qf_all + warp * (A::Q_BYTES / 16);
    uint32_t phase = 0;  // bit 0: of the warp's first barrier, bit 1: of its second one
    bool ok = true;
    auto group_sync = [&] {  // (barrier numbers as constants: a number in a register takes all sixteen)
        if (group == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
        else asm volatile("bar.sync 2, 128;" ::: "memory");
    };
    for (int i = group; i < n_tok; i += 2) {
        const uint32_t seq = sh.seq[i], len = sh.pos[i] + 1u;
        if (len <= p0) continue;
        const size_t head_row = (size_t)(t_lo + i) * p.n_q_heads + (size_t)h * gsize;
        float m = -INFINITY, l = 0.0f;
        if (p0 + (uint32_t)(wl * PM_TILE) < len && ok) {
            const uint32_t blocks = at_blocks(p, seq, len, p0, lane);
            uint32_t live = at_load_tile<HD>(p, &maps.k, blocks, len, h, p0, wl, tile_k, bar, lane, seq);
            if (BOTH) at_load_tile<HD>(p, &maps.v, blocks, len, h, p0, wl, tile_v, bar + 8u, lane, seq);
            at_load_q<HD>(g < gsize ? p.q + (head_row + g) * HD : nullptr, nullptr, 0, p.scale, qf, lane);
            ok = ts_wait(bar, phase & 1u);
            ok = __all_sync(0xffffffffu, ok);
            phase ^= 1u;
            if (ok) {
                uint32_t phi[4], plo[4];
                at_scores<HD>(rows, tile_k, qf, live, lane, phi, plo, m, l);
                __syncwarp();
                if (!BOTH) live = at_load_tile<HD>(p, &maps.v, blocks, len, h, p0, wl, tile_v, bar, lane, seq);
                ok = BOTH ? ts_wait(bar + 8u, (phase >> 1) & 1u) : ts_wait(bar, phase & 1u);
                ok = __all_sync(0xffffffffu, ok);
                phase ^= BOTH ? 2u : 1u;
                if (live != 0xffffffffu) at_zero_rows<HD>(rows, tile_v, live, lane);
                __syncwarp();
                float acc[A::NT][2];
#pragma unroll
                for (int k = 0; k < A::NT; ++k) acc[k][0] = acc[k][1] = 0.0f;
                at_pv<HD>(rows, tile_v, phi, plo, 1.0f, lane, acc);
                if (live != 0xffffffffu) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                // (the query's fragments are done with: their place takes the warp's eight rows)
                float *to = (float *)qf + g * HD + 2 * tq;
                if (g < gsize) {
#pragma unroll
                    for (int k = 0; k < A::NT; ++k) *(float2 *)(to + 8 * k) = make_float2(acc[k][0], acc[k][1]);
                }
            }
        }
        if (tq == 0) sh.m[warp][g] = ok ? m : -INFINITY, sh.l[warp][g] = l;
        group_sync();
        for (int k = wl * 32 + lane; k < gsize * HD; k += 128) {
            const int hh = k / HD, d = k % HD;
            float M = -INFINITY, L = 0.0f, O = 0.0f;
#pragma unroll
            for (int w = 0; w < 4; ++w) M = fmaxf(M, sh.m[4 * group + w][hh]);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float mw = sh.m[4 * group + w][hh];
                if (M == -INFINITY || mw == -INFINITY) continue;
                const float e = expf(mw - M);
                L += sh.l[4 * group + w][hh] * e;
                O += ((const float *)(qf_all + (4 * group + w) * (A::Q_BYTES / 16)))[k] * e;
            }
            if (len <= (uint32_t)PM_CHUNK || n_chunks == 1) {
                p.out[(head_row + hh) * HD + d] = L > 0.0f ? O / L : 0.0f;
                continue;
            }
            float *pr = partial + ((head_row + hh) * n_chunks + c) * (HD + 2);
            if (d == 0) *(float2 *)pr = make_float2(M, L);
            pr[2 + d] = O;
        }
        group_sync();
    }
    return ok;
}

// Prompts: the tokens' K and V rows are in the pool, q is rotated.  grid (KV heads, blocks of tokens, chunks).
template <int HD>
__global__ void __launch_bounds__(32 * AT_WARPS, 2)
attention_prompt_kernel(const __grid_constant__ AttnMaps maps, PagedParams p, int block_tokens, int n_chunks, float *partial, int *err) {
    using A = At<HD>;
    extern __shared__ uint8_t at_smem[];
    __shared__ AtPromptShared sh;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), g = lane >> 2, tq = lane & 3;
    const uint32_t raw = tm_smem_u32(at_smem), base = (raw + 1023u) & ~1023u;
    uint4 *qf_all = (uint4 *)(at_smem + (base - raw) + A::PROMPT_TILES * A::TILE), *qf = qf_all + warp * (A::Q_BYTES / 16);
    const uint32_t bar = tm_smem_u32(&sh.bars[warp][0]);
    if (lane == 0) {
        tm_mbar_init(bar, 1);
        tm_mbar_init(bar + 8u, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    uint32_t *s_seq = sh.seq, *s_pos = sh.pos, *tile_live = sh.tile_live;
    const int odd_v = *p.odd_v;
    const int h = blockIdx.x, c = blockIdx.z, t_lo = blockIdx.y * block_tokens, n_tok = min(block_tokens, p.n_tokens - t_lo);
    const int H = p.n_kv_heads, gsize = p.n_q_heads / H, per_pass = 8 / gsize;
    const AtRows<HD> rows{min(p.block_shift, 5)};
    const uint32_t p0 = (uint32_t)c * PM_CHUNK;
    if (threadIdx.x < (unsigned)n_tok) {
        s_seq[threadIdx.x] = p.meta[(t_lo + threadIdx.x) * 4];
        s_pos[threadIdx.x] = p.meta[(t_lo + threadIdx.x) * 4 + 1];
    }
    __syncthreads();
    // A run: tokens of one sequence at consecutive positions.  Blocks whose runs are short are taken token by token, and so is everything
    // where a V value of the call is not finite: a run's tokens share the V rows of its longest context, and a token's zero
    // probability times such a value beyond its own context would be NaN.
    bool ok = true;
    uint32_t phase = 0;
    const int n_runs = __popc(__ballot_sync(0xffffffffu, lane < n_tok && (lane == 0 || s_seq[lane] != s_seq[lane - 1] || s_pos[lane] != s_pos[lane - 1] + 1u)));
    const bool by_token = (n_tok < AT_SHORT * n_runs && (n_runs > 1 || n_tok == 1)) || odd_v != 0;
    if (by_token) {
        if (!at_tokens<HD>(maps, p, t_lo, n_tok, h, c, n_chunks, partial, base, qf_all, sh)) {
            if (lane == 0) atomicExch(err, 61);
            for (int i = 0; i < 200; ++i) __nanosleep(1000);
        }
        return;
    }
    for (int first = 0, n = 1; first < n_tok; first += n) {
        const uint32_t seq = s_seq[first], pos = s_pos[first];
        for (n = 1; first + n < n_tok && s_seq[first + n] == seq && s_pos[first + n] == pos + (uint32_t)n; ++n) {}
        const uint32_t len = pos + (uint32_t)n;  // the longest context
        if (len <= p0) continue;
        __syncthreads();  // the tiles of the run before have been read
        {
            const uint32_t tile = base + (uint32_t)(warp * A::TILE);
            uint32_t live = 0u;
            if (p0 + (uint32_t)((warp & 3) * PM_TILE) < len)
                live = at_load_tile<HD>(p, warp < 4 ? &maps.k : &maps.v, at_blocks(p, seq, len, p0, lane), len, h, p0, warp & 3, tile, bar, lane, seq);
            else if (lane == 0) tm_mbar_arrive(bar);
            if (lane == 0) tile_live[warp] = live;
            ok = ok && ts_wait(bar, phase);
            ok = __all_sync(0xffffffffu, ok);
            phase ^= 1u;
            if (warp >= 4 && live != 0xffffffffu) {
                at_zero_rows<HD>(rows, tile, live, lane);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
        }
        if (__syncthreads_or(!ok)) break;
        for (int sub = warp * per_pass; sub < n; sub += AT_WARPS * per_pass) {
            // row g of A: query head g % gsize of token g / gsize of the pass
            const int tok = g / gsize, last = min(sub + per_pass, n);  // of the pass
            const bool row_ok = tok < per_pass && sub + tok < n;
            const int t = t_lo + first + sub + (row_ok ? tok : 0);
            const uint32_t row_len = s_pos[t - t_lo] + 1u, most = pos + (uint32_t)last;  // context of the row's token; the longest
            if (most <= p0) continue;
            // (32 bits, as the warp number is one per warp: what else is kept spills; 9 tokens in each of 64 sequences of 2000 439 us, 409 so)
            const int row = t * p.n_q_heads + h * gsize + (row_ok ? g - tok * gsize : 0);
            at_load_q<HD>(row_ok ? p.q + (size_t)row * HD : nullptr, nullptr, 0, p.scale, qf, lane);
            AtTiles tiles;
            float M, L;
#pragma unroll 1
            for (int w = 0; w < 4; ++w) {
                const uint32_t k0 = p0 + (uint32_t)w * PM_TILE;
                tiles.push();
                if (k0 >= most) continue;
                const uint32_t row_live = row_len <= k0 ? 0u : tile_live[w] & (row_len - k0 >= 32u ? 0xffffffffu : (1u << (row_len - k0)) - 1u);
                at_scores<HD>(rows, base + (uint32_t)(w * A::TILE), qf, row_live, lane, tiles.phi[0], tiles.plo[0], tiles.m[0], tiles.l[0]);
            }
            tiles.weigh(M, L);
            float acc[A::NT][2];
#pragma unroll
            for (int k = 0; k < A::NT; ++k) acc[k][0] = acc[k][1] = 0.0f;
#pragma unroll 1
            for (int w = 0; w < 4 && p0 + (uint32_t)w * PM_TILE < most; ++w, tiles.shift())
                at_pv<HD>(rows, base + (uint32_t)((4 + w) * A::TILE), tiles.phi[3], tiles.plo[3], tiles.l[3], lane, acc);
            if (row_ok && row_len > p0)
                at_store<HD>(p, partial, n_chunks, row, c, row_len <= (uint32_t)PM_CHUNK || n_chunks == 1, M, L, tq, acc);
        }
    }
    if (!ok) {
        if (lane == 0) atomicExch(err, 61);
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
}

// ---- host ----
// [slabs of block_size rows][64 dimensions][rows][dimensions]; how many slabs the pool has is not known here, and no box is asked for outside it
static cudaError_t at_encode(CUtensorMap *m, const void *pool, int head_dim, int block_shift) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (encode == nullptr) return cudaErrorNotSupported;
    const cuuint64_t bs = (cuuint64_t)1 << block_shift;
    const cuuint64_t row = (cuuint64_t)head_dim * 2, halves = (cuuint64_t)head_dim / 64;
    const cuuint64_t dims[4] = {64u, bs, halves, 0x7fffffffu}, strides[3] = {row, 128u, bs * row};
    const cuuint32_t box[4] = {64u, (cuuint32_t)(bs < PM_TILE ? bs : PM_TILE), (cuuint32_t)halves, 1u}, step[4] = {1u, 1u, 1u, 1u};
    const CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(pool), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
template <typename... KArgs, typename... Args>
static cudaError_t at_launch(void (*kernel)(KArgs...), dim3 grid, size_t smem, cudaStream_t s, Args... args) {
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(32 * AT_WARPS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    static const bool no_pdl = getenv("MARMOT_CUDA_NO_PDL") != nullptr;  // diagnostic switch
    cfg.numAttrs = no_pdl ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
static cudaError_t at_maps(const PagedParams &p, int head_dim, AttnMaps &maps) {
    if (cudaError_t e = at_encode(&maps.k, p.kv_k, head_dim, p.block_shift)) return e;
    return at_encode(&maps.v, p.kv_v, head_dim, p.block_shift);
}

// Heads of 64 stay with paged_attention_mma_kernel: its small CTAs keep seven chunks of four warps on an SM, and a tile is too short to
// pay for a warp's turn here (32 sequences of 1000, 16 heads of 64: 33 us there, 48 here; 32 heads on 8 of 128: 44 and 41).
bool attention_decode_supported(int n_tokens, int head_dim) { return n_tokens <= AT_MAX_TOKENS && head_dim == 128; }

cudaError_t launch_attention_decode(const PagedParams &p, int n_chunks, float *partial, const FusedDecode &fd, int *err,
                                    cudaStream_t s) {
    AttnMaps maps;
    if (cudaError_t e = at_maps(p, 128, maps)) return e;
    const long warps = (long)p.n_tokens * p.n_kv_heads * n_chunks, most = device_sm_count();
    const long ctas = (warps + AT_WARPS - 1) / AT_WARPS;
    const dim3 grid((unsigned)(ctas < most ? ctas : most));
    return at_launch(attention_decode_kernel<128>, grid, 1024 + AT_WARPS * (AT_RING_BYTES + At<128>::Q_BYTES), s, maps, p, n_chunks, partial, fd, err);
}

cudaError_t launch_attention_prompt(const PagedParams &p, int head_dim, int n_chunks, float *partial, int *err, cudaStream_t s) {
    AttnMaps maps;
    if (cudaError_t e = at_maps(p, head_dim, maps)) return e;
    // As many tokens per CTA as leave two CTAs per SM, counting the chunks of the longest context that the block table allows: the
    // more, the fewer copies of K and V from L2; but a CTA takes its tokens of different sequences one after the other.
    int block = AT_BLOCK;
    while (block > 1 && (long)p.n_kv_heads * n_chunks * ((p.n_tokens + block - 1) / block) < 2l * device_sm_count()) block /= 2;
    const dim3 grid((unsigned)p.n_kv_heads, (unsigned)((p.n_tokens + block - 1) / block), (unsigned)n_chunks);
    auto bytes = [](int tiles, int tile, int q) { return (size_t)(1024 + tiles * tile + AT_WARPS * q); };
    const size_t smem = head_dim == 64 ? bytes(At<64>::PROMPT_TILES, At<64>::TILE, At<64>::Q_BYTES) : bytes(At<128>::PROMPT_TILES, At<128>::TILE, At<128>::Q_BYTES);
    return head_dim == 64 ? at_launch(attention_prompt_kernel<64>, grid, smem, s, maps, p, block, n_chunks, partial, err)
                          : at_launch(attention_prompt_kernel<128>, grid, smem, s, maps, p, block, n_chunks, partial, err);
}

}  // namespace mcu
